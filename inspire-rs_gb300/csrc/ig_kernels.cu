// Kernels of the InspiRING respond path on sm_103a.
//
// Work map (reference call sites in src/):
//   key_rows      the seat's key body (pir/session.rs:600-625) and the offline mask rows
//                 (inspiring/inspiring2.rs:537-598) transformed, folded and scaled once.
//   ntt_rows      negacyclic forward NTT of many rows (Galois keys, the client's secret).
//   store_ntt     a shard's columns transformed before its store is folded
//                 (inspiring/shard_store.rs:139-144).
//   store_fold    step 1 of the offline phase folded over one shard's columns
//                 (inspiring/inspiring2.rs:964-1004 via shard_store.rs:145), computed per
//                 slot as a length-gamma cyclic DFT instead of gamma^2 monomial products.
//   shard_scan    the store's column check and b fold (shard_store.rs:197-264): one HBM
//                 pass over the queried shard's columns per query.
//   respond       one CTA, or a cluster of two or four, per query: the `a` expansion (math/poly.rs:657-686),
//                 the store gather (shard_store.rs:282-342), the backward recursion
//                 (inspiring2.rs:1014-1085) with the online gather fused into each link
//                 (inspiring2.rs:1393-1485), the final inverse transforms and the 36-bit
//                 mod switch (pir/mod_switch.rs:148-176).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "ig_inbox.cuh"
#include "ig_kernels.cuh"

namespace igk {
using namespace ig;

// ------------------------------------------------------------------------------------
// Negacyclic transforms in shared memory. Forward: Cooley-Tukey over the bit-reversed
// ladder psi^brv(m) (math/ntt.rs:600-623 order); inverse: Gentleman-Sande over the
// inverse ladder (math/ntt.rs:626-654) without the final n^-1, which consumers fold into
// their first use. Both are linear in standard form.
//
// Radix-4 transforms: each thread carries one 4-element unit through two consecutive stages in
// registers (N/4 threads), halving shared-memory round trips and barriers against a
// stage-per-barrier radix-2 schedule. Odd log n adds one radix-2 stage (first in the forward,
// last in the inverse). Words are lazy: a product by a twiddle (mulw) lands in [0, 2q + 2^47) for
// any 64-bit operand, so a 64-bit word has room for 16q of sums and a word is brought back to
// just above q (red60) only where the next sums could pass that. Bounds are written beside each
// pass in units of q; "2+" is a little above 2q.

// Forward butterfly (Cooley-Tukey): X grows by at most 3q, Y is any 64-bit word.
__device__ __forceinline__ void bf_fwd(u64& X, u64& Y, const Tw& w) {
  const u64 t = mulw(Y, w);
  Y = X - t + 3 * Q;
  X += t;
}

// Inverse butterfly (Gentleman-Sande), X, Y -> X + Y, (X - Y) w^-1, with the forward ladder's
// entry f of the mirrored index: w^-1 = psi^-brv(m) = -f, so (X - Y) w^-1 = (Y - X) f, and
// f = ladder[3 2^s - 1 - m] for m in [2^s, 2^(s+1)). X must be at most C q.
template <int C>
__device__ __forceinline__ void bf_inv(u64& X, u64& Y, const Tw& f) {
  const u64 d = Y - X + C * Q;
  X += Y;
  Y = mulw(d, f);
}

// Two forward stages on a unit; out <= in + 6. RED brings the two words that are not multiplied
// first down to 1, and the outputs are then at most 7.
template <bool RED>
__device__ __forceinline__ void fwd_unit(u64& a0, u64& a1, u64& a2, u64& a3, const Tw& wa, const Tw& wb,
                                         const Tw& wc) {
  if (RED) {
    a0 = red60(a0);
    a1 = red60(a1);
  }
  bf_fwd(a0, a2, wa);
  bf_fwd(a1, a3, wa);
  bf_fwd(a0, a1, wb);
  bf_fwd(a2, a3, wc);
}

// Two inverse stages on a unit of words up to 2+: sums up to 8+ and 4+ come back to 1, products
// are 2+.
__device__ __forceinline__ void inv_unit(u64& a0, u64& a1, u64& a2, u64& a3, const Tw& f0, const Tw& f1,
                                         const Tw& f2) {
  bf_inv<3>(a0, a1, f0);
  bf_inv<3>(a2, a3, f1);
  bf_inv<5>(a0, a2, f2);
  bf_inv<3>(a1, a3, f2);
  a0 = red60(a0);
  a1 = red60(a1);
}

// In: at most 2. Out: at most 7.
template <int LOGN, int NT, int NB>
__device__ __forceinline__ void ntt_fwd_r4(u64* const (&x)[NB], const Tw* tw) {
  constexpr int N = 1 << LOGN, UPT = N / 4 / NT;
  static_assert(UPT >= 1 && (N / 4) % NT == 0, "whole radix-4 units per thread");
  const int tid = threadIdx.x;
  int s = 0;
  if (LOGN & 1) {
    constexpr int t = N / 2;
    const Tw w = tw[1];
#pragma unroll
    for (int r = 0; r < 2 * UPT; r++) {
      const int b = tid + r * NT;
#pragma unroll
      for (int k = 0; k < NB; k++) {
        u64 a = x[k][b], c = x[k][b + t];
        bf_fwd(a, c, w);
        x[k][b] = a;
        x[k][b + t] = c;
      }
    }
    __syncthreads();
    s = 1;
  }
#pragma unroll 1
  for (; s < LOGN; s += 2) {
    const int t = N >> (s + 1), m = 1 << s, h = t >> 1;
#pragma unroll
    for (int uu = 0; uu < UPT; uu++) {
      const int u = tid + uu * NT;
      const int i = u / h, o = u - i * h;
      const int e0 = i * 2 * t + o;
      const Tw wa = tw[m + i], wb = tw[2 * m + 2 * i], wc = tw[2 * m + 2 * i + 1];
#pragma unroll
      for (int k = 0; k < NB; k++) {
        u64 a0 = x[k][e0], a1 = x[k][e0 + h], a2 = x[k][e0 + t], a3 = x[k][e0 + t + h];
        fwd_unit<true>(a0, a1, a2, a3, wa, wb, wc);
        x[k][e0] = a0;
        x[k][e0 + h] = a1;
        x[k][e0 + t] = a2;
        x[k][e0 + t + h] = a3;
      }
    }
    __syncthreads();
  }
}

// In: at most 2+. Out: at most 4+, without n^-1.
template <int LOGN, int NT, int NB>
__device__ __forceinline__ void ntt_inv_r4(u64* const (&x)[NB], const Tw* tw) {
  constexpr int N = 1 << LOGN, UPT = N / 4 / NT;
  static_assert(UPT >= 1 && (N / 4) % NT == 0, "whole radix-4 units per thread");
  const int tid = threadIdx.x;
  int s = 0;
#pragma unroll 1
  for (; s + 1 < LOGN; s += 2) {
    const int t = 1 << s, m = N >> (s + 1);
#pragma unroll
    for (int uu = 0; uu < UPT; uu++) {
      const int u = tid + uu * NT;
      const int B = u >> s, o = u & (t - 1);
      const int e0 = B * 4 * t + o;
      const Tw f0 = tw[2 * m - 1 - 2 * B], f1 = tw[2 * m - 2 - 2 * B], f2 = tw[m - 1 - B];
#pragma unroll
      for (int k = 0; k < NB; k++) {
        u64 a0 = x[k][e0], a1 = x[k][e0 + t], a2 = x[k][e0 + 2 * t], a3 = x[k][e0 + 3 * t];
        inv_unit(a0, a1, a2, a3, f0, f1, f2);
        x[k][e0] = a0;
        x[k][e0 + t] = a1;
        x[k][e0 + 2 * t] = a2;
        x[k][e0 + 3 * t] = a3;
      }
    }
    __syncthreads();
  }
  if (LOGN & 1) {
    constexpr int t = N / 2;
    const Tw f = tw[1];
#pragma unroll
    for (int r = 0; r < 2 * UPT; r++) {
      const int b = tid + r * NT;
#pragma unroll
      for (int k = 0; k < NB; k++) {
        u64 a = x[k][b], c = x[k][b + t];
        bf_inv<3>(a, c, f);
        x[k][b] = a;
        x[k][b + t] = c;
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------
// Batched forward NTT: one CTA per row.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_ntt_rows(CrsDev c, const u64* in, u64* out, Tw scale) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  Tw* tw = reinterpret_cast<Tw*>(sm);
  u64* x = sm + 2 * N;
  const u64* row = in + (size_t)blockIdx.x * N;
  for (int k = threadIdx.x; k < N; k += NT) {
    x[k] = reduce128(row[k]);
    tw[k] = c.tw[k];
  }
  __syncthreads();
  {
    u64* const bufs[1] = {x};
    ntt_fwd_r4<LOGN, NT, 1>(bufs, tw);
  }
  u64* o = out + (size_t)blockIdx.x * N;
  for (int k = threadIdx.x; k < N; k += NT) o[k] = canon(mulw(x[k], scale));
}

// ------------------------------------------------------------------------------------
// Store fold. For slot t with root w_t = w0^e_t, step 1 at rotation i reads
//   acc_i[t] = sum_j w_t^(j * c_i) H_j[t],  c_i = g^-i mod 2n = 1 + m_i * (2n/gamma),
// so with u_j = w0^(e_t j) H_j[t] and zeta = w0^(2n/gamma) (order gamma),
//   acc_i[t] = DFT_zeta(u)[(e_t * m_i) mod gamma].
// The sum lands at S_i[t'] with table_i[t'] = t, i.e. t' = slot of exponent c_i * e_t,
// scaled by gamma^-1 and stored in R-form.
//
// One launch folds several shards (blockIdx.y): a shard alone leaves most of the GPU idle. What bounds it is the LSU
// path, so its gathers are few: slot t = 8u + k of a unit has e_t = e_8u + brv3(k) 2n/8, so a unit's words share the
// power w0^(e_8u j), one load for its lanes, and take one of eight multiples of it from shared memory (fold_unit); the slot
// table is staged; the twiddles of a pass lie side by side; fold_sw spreads the words of every pass over the banks.
// Powers gathered a word, twiddles a stride apart and divisions by the runtime tile: 61 us for eight shards of gamma 256.
constexpr int FOLD_TILE_LOG = 11, FOLD_TILE = 1 << FOLD_TILE_LOG;
constexpr int FOLD_THREADS = 256;

// The shard a store kernel works on: entry blockIdx.y of a device table, or the one given.
struct ShardArg {
  const ShardDev* table;
  ShardDev one;
};
__device__ __forceinline__ ShardDev shard_of(const ShardArg& a) { return a.table ? a.table[blockIdx.y] : a.one; }

__device__ __forceinline__ u32 fold_sw(u32 e) { return e ^ (((e >> 4) & 3) * 5); }
// Twiddles of a fold of length gamma: len entries a pass of two stages.
__host__ __device__ constexpr u32 fold_twiddles(u32 gamma) {
  u32 n = 0;
  for (u32 len = gamma >> 1; len >= 2; len >>= 2) n += len;
  return n;
}

// LG = log gamma; lgs = log SL, which the tile fixes from gamma 8 up.
template <int LG>
__global__ void __launch_bounds__(FOLD_THREADS) k_store_fold(CrsDev c, const u64* H, ShardArg shards, u32 lgs_) {
  constexpr u32 gamma = 1u << LG, half = gamma >> 1, row = gamma + 1, BATCH = 4;
  const u32 lgs = LG >= 3 ? FOLD_TILE_LOG - LG : lgs_, SL = 1u << lgs, n = c.n, m2n = 2 * n - 1;
  const u32 tile = SL * gamma;  // SL slots per CTA, tile <= FOLD_TILE words
  extern __shared__ __align__(16) u64 sm[];
  Tw* zeta = reinterpret_cast<Tw*>(sm);
  Tw* unit = zeta + fold_twiddles(gamma);
  uint16_t* slots = reinterpret_cast<uint16_t*>(unit + 8);
  u64* x = reinterpret_cast<u64*>(slots + n);  // [slot][fold_sw(j)], a word of padding per slot
  const u32 t0 = blockIdx.x * SL, tid = threadIdx.x;
  H += ((size_t)blockIdx.y * gamma << c.logn) + t0;
  u64* sums = const_cast<u64*>(shard_of(shards).sums_R);
  for (u32 k = tid; k < n / 8; k += FOLD_THREADS)
    reinterpret_cast<uint4*>(slots)[k] = reinterpret_cast<const uint4*>(c.exp_slot)[k];
  if (tid < 8) unit[tid] = c.fold_unit[tid];
#pragma unroll
  for (u32 len = half, at = 0; len >= 2; at += len, len >>= 2)
    for (u32 k = tid; k < len; k += FOLD_THREADS) zeta[at + k] = c.zeta[k * (half / len)];
  __syncthreads();
#pragma unroll
  for (u32 i0 = tid; i0 < tile; i0 += BATCH * FOLD_THREADS) {
    u64 h[BATCH];
    Tw w[BATCH];
#pragma unroll
    for (u32 r = 0; r < BATCH; r++) {
      const u32 idx = i0 + r * FOLD_THREADS, j = idx >> lgs, s = idx & (SL - 1);
      if (idx >= tile) break;
      h[r] = H[(j << c.logn) + s];
      w[r] = c.pow_root[(c.slot_exp[(t0 + s) & ~7u] * j) & m2n];
    }
#pragma unroll
    for (u32 r = 0; r < BATCH; r++) {
      const u32 idx = i0 + r * FOLD_THREADS, j = idx >> lgs, s = idx & (SL - 1);
      if (idx >= tile) break;
      const u32 k = (__brev((t0 + s) & 7) >> 29) * j & 7;
      x[s * row + fold_sw(j)] = mulw(mulw(h[r], w[r]), unit[k]);
    }
  }
  __syncthreads();
  // Gentleman-Sande DFT of length gamma per slot, bit-reversed output, two stages a pass on words up to
  // 2+ (sums up to 8+ and 4+ reduced, products 2+), a last stage alone when log gamma is odd.
  const Tw* z = zeta;
#pragma unroll
  for (u32 len = half; len >= 2; z += len, len >>= 2) {
    const u32 q = len >> 1;
#pragma unroll 2
    for (u32 b = tid; b < tile / 4; b += FOLD_THREADS) {
      const u32 s = b / (gamma / 4 ? gamma / 4 : 1), bb = b & (gamma / 4 - 1);
      const u32 j = bb & (q - 1), i0 = (bb - j) * 4 + j;
      u64* y = x + s * row;
      const u32 e0 = fold_sw(i0), e1 = fold_sw(i0 + q), e2 = fold_sw(i0 + len), e3 = fold_sw(i0 + len + q);
      u64 a0 = y[e0], a1 = y[e1], a2 = y[e2], a3 = y[e3];
      const u64 s0 = a0 + a2, s1 = a1 + a3;
      const u64 d0 = mulw(a0 - a2 + 3 * Q, z[j]), d1 = mulw(a1 - a3 + 3 * Q, z[j + q]);
      const Tw w = z[2 * j];
      y[e0] = red60(s0 + s1);
      y[e1] = mulw(s0 - s1 + 5 * Q, w);
      y[e2] = red60(d0 + d1);
      y[e3] = mulw(d0 - d1 + 3 * Q, w);
    }
    __syncthreads();
  }
  if constexpr (LG & 1) {
    for (u32 b = tid; b < tile / 2; b += FOLD_THREADS) {
      u64* y = x + b / half * row;
      const u32 i0 = 2 * (b & (half - 1)), e0 = fold_sw(i0), e1 = fold_sw(i0 + 1);
      const u64 u = y[e0], v = y[e1];
      y[e0] = u + v;
      y[e1] = u - v + 3 * Q;
    }
    __syncthreads();
  }
#pragma unroll 4
  for (u32 idx = tid; idx < tile; idx += FOLD_THREADS) {
    const u32 i = idx >> lgs, s = idx & (SL - 1);
    const u32 e = c.slot_exp[t0 + s];
    const u32 k = (e * c.m_of_i[i]) & (gamma - 1);
    const u32 kr = LG ? __brev(k) >> (32 - (LG ? LG : 1)) : 0;
    const u32 tp = slots[((c.cpow[i] * e) & m2n) >> 1];
    sums[((size_t)i << c.logn) + tp] = canon(x[s * row + fold_sw(kr)]);
  }
}

// ------------------------------------------------------------------------------------
// Shard scan (shard_store.rs:197-264), split in two.
//
// Column tags (k_column_tags). Per word w_k of column j:
//   tag = sum_k lo32(w_k) key[2k] + hi32(w_k) key[2k+1]   (mod 2^61 - 1)
// The reference recomputes the tags from the caller's columns at every respond and refuses
// a shard whose columns no longer give the stored tags. Here the columns live in device
// memory the library owns and change only through its own calls (a shard upload or an
// encode), so the tags are recomputed once, at each such change, and compared with the
// stored ones: a mismatch marks the shard stale, and every later respond on it is refused
// with the reference's message until the store is rebuilt. The refusal stays at respond
// time; the tag check leaves the per-query scan. A launch covers a range of shards, and those of
// them that hold no store have no tag key and no tags: their CTAs return at once.
//
// b fold (k_scan), per query and column j of its shard:
//   fold_j = sum_k w_k * b_rev[k],  b_rev[0] = b_0, b_rev[k] = -b_{n-k}   (mod q)
// = coeff0(b * h_j). Compact shards (every word below 2^16, kept as a u16 copy): the fold
// is a matrix-vector product of the column words with b_rev, whose words are split into
// two 32-bit limbs and staged once per CTA in shared memory. Every product w * limb is
// below 2^48, so a lane's 64-bit accumulators hold its 64 products per column exactly, and
// the limbs recombine into a 128-bit sum at the end: two 32x32->64 multiply-adds per
// 16-bit word. The vector layout V[k & 7][k >> 3] lets lane l read positions 8m..8m+7
// (m = l + 32 it) conflict-free while it reads the same positions of a column as one
// 16-byte word. Other shards take an exact 128-bit path over the u64 words.
//
// Work items: a CTA takes SCAN_COLS consecutive columns of one query (SCAN_ROWS per warp),
// item = query << 12 | chunk from a per-launch list, so queries of different widths share
// a launch; without a list CTA b takes query b / chunks, chunk b % chunks.
constexpr int SCAN_WARPS = 16;
constexpr int SCAN_ROWS = 4;
constexpr int SCAN_COLS = SCAN_WARPS * SCAN_ROWS;
constexpr int SCAN_STAGES = 2;
constexpr u64 TAG_PRIME = (1ULL << 61) - 1;

__device__ __forceinline__ u128 shfl_xor_u128(u128 v, int m) {
  u64 lo = (u64)v, hi = (u64)(v >> 64);
  lo = __shfl_xor_sync(0xffffffffu, lo, m);
  hi = __shfl_xor_sync(0xffffffffu, hi, m);
  return ((u128)hi << 64) | lo;
}

__device__ __forceinline__ u64 tag_residue(u128 tag) {
  u128 t = (tag & TAG_PRIME) + (tag >> 61);
  t = (t & TAG_PRIME) + (t >> 61);
  u64 tv = (u64)t;
  while (tv >= TAG_PRIME) tv -= TAG_PRIME;
  return tv;
}
// Writes column j's tag, or with a mismatch word given compares it with the stored one.
__device__ __forceinline__ void put_tag(const ShardDev& sh, u32 j, u64 tag, u32* mismatch) {
  if (!mismatch)
    const_cast<u64*>(sh.tags)[j] = tag;
  else if (tag != sh.tags[j])
    atomicOr(mismatch + blockIdx.y, 1u);
}

// A shard's tag key: 2n words below 2^61 - 1 from the ChaCha20 keystream of a seed drawn from OS entropy
// (shard_store.rs:127-135), stream `stream` + the shard's place in the launch. A candidate at the bound
// (probability 2^-61) gives way to the same word of the streams 2^32 further on.
struct TagSeed {
  u32 w[8];
};
__global__ void k_tag_keys(u32 n, const ShardDev* table, TagSeed seed, u64 stream) {
  const u32 b = blockIdx.x * blockDim.x + threadIdx.x;  // one block of eight words
  if (b >= n / 4) return;
  u64* key = const_cast<u64*>(table[blockIdx.y].tag_key) + 8 * (size_t)b;
  u32 blk[16];
  chacha20_block(seed.w, b, stream + blockIdx.y, blk);
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    u64 v = (((u64)blk[2 * k + 1] << 32) | blk[2 * k]) >> 3;
    for (u64 more = 1; v >= TAG_PRIME && more < 64; more++) {
      u32 alt[16];
      chacha20_block(seed.w, b, stream + blockIdx.y + (more << 32), alt);
      v = (((u64)alt[2 * k + 1] << 32) | alt[2 * k]) >> 3;
    }
    key[k] = v;
  }
}

// Tags of the columns of wide shards (words of 2^16 and above): one warp per column.
template <int LOGN>
__global__ void __launch_bounds__(256) k_column_tags(u32 gamma, const ShardDev* table, u32* mismatch) {
  constexpr int N = 1 << LOGN;
  const ShardDev sh = table[blockIdx.y];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const u32 j = blockIdx.x * (blockDim.x >> 5) + warp;
  if (j >= gamma || sh.cols16 || !sh.tag_key) return;
  const u64* col = sh.columns + (size_t)j * N;
  u128 tag = 0;
#pragma unroll 4
  for (int k = lane; k < N; k += 32) {
    const u64 w = col[k];
    const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(sh.tag_key + 2 * k);
    tag += (u128)(w & 0xffffffffULL) * kk.x + (u128)(w >> 32) * kk.y;
  }
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) tag += shfl_xor_u128(tag, m);
  if (lane == 0) put_tag(sh, j, tag_residue(tag), mismatch);
}

// Shared memory of the compact path: the vector V, then per warp a ring of SCAN_STAGES
// steps of column chunks its lanes copy ahead (cp.async), so the next steps' loads are in
// flight while the current step's products run.
__host__ __device__ constexpr size_t scan_smem_bytes(int n) {
  return (size_t)n * 8 + (size_t)SCAN_WARPS * SCAN_STAGES * SCAN_ROWS * 32 * 16;
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(addr), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory");
}

// Sums eight per-lane values over the warp in nine 64-bit exchanges instead of forty:
// each step halves the values a lane keeps and doubles the lanes summed into them. On
// return, lane l holds the warp total of value ((l >> 4) & 1) * 4 + ((l >> 3) & 1) * 2 +
// ((l >> 2) & 1) in v[0].
__device__ __forceinline__ void warp_reduce8(u64 (&v)[8], int lane) {
  {
    const bool up = lane & 16;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const u64 send = up ? v[k] : v[k + 4];
      const u64 got = __shfl_xor_sync(0xffffffffu, send, 16);
      v[k] = (up ? v[k + 4] : v[k]) + got;
    }
  }
  {
    const bool up = lane & 8;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const u64 send = up ? v[k] : v[k + 2];
      const u64 got = __shfl_xor_sync(0xffffffffu, send, 8);
      v[k] = (up ? v[k + 2] : v[k]) + got;
    }
  }
  {
    const bool up = lane & 4;
    const u64 send = up ? v[0] : v[1];
    const u64 got = __shfl_xor_sync(0xffffffffu, send, 4);
    v[0] = (up ? v[1] : v[0]) + got;
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Sums word_k v_k over `rows` (at most SCAN_ROWS) columns at col for a vector of 64-bit words v: fill(V)
// writes v's 32-bit limbs (shared by the CTA's warps, V[k & 7][k >> 3]) while the warp's first copies are
// in flight, out(r, sum) gets row r's 128-bit sum on one lane. All the CTA's threads call it.
template <int LOGN, class Fill, class Out>
__device__ __forceinline__ void scan_columns16(uint4* scan_sm, const uint16_t* col, int rows, Fill fill, Out out) {
  constexpr int N = 1 << LOGN, M = N / 8, ITER = M / 32;
  uint2* V = reinterpret_cast<uint2*>(scan_sm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint4* ring = scan_sm + N / 2 + (size_t)warp * SCAN_STAGES * SCAN_ROWS * 32;
  // Lane l copies, for step it, the 16-byte chunk at positions 8m..8m+7 (m = l + 32 it)
  // of each of the warp's rows into its own ring slots.
  auto issue = [&](int it) {
    if (it < ITER) {
      uint4* dst = ring + (it % SCAN_STAGES) * SCAN_ROWS * 32 + lane;
      const int m = lane + 32 * it;
      for (int r = 0; r < rows; r++) cp_async16(dst + r * 32, col + (size_t)r * N + 8 * m);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int it = 0; it < SCAN_STAGES - 1; it++) issue(it);
  fill(V);
  __syncthreads();
  if (rows == 0) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    return;
  }
  u64 acc[8];  // acc[2r] = low-limb sum of row r, acc[2r + 1] = high-limb sum
#pragma unroll
  for (int k = 0; k < 8; k++) acc[k] = 0;
#pragma unroll 1
  for (int it = 0; it < ITER; it++) {
    issue(it + SCAN_STAGES - 1);
    cp_async_wait<SCAN_STAGES - 1>();  // step it's copies have landed
    const int m = lane + 32 * it;
    const uint4* src = ring + (it % SCAN_STAGES) * SCAN_ROWS * 32 + lane;
    uint4 w[SCAN_ROWS];
#pragma unroll
    for (int r = 0; r < SCAN_ROWS; r++) w[r] = r < rows ? src[r * 32] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int p = 0; p < 8; p++) {
      const uint2 v = V[p * M + m];
#pragma unroll
      for (int r = 0; r < SCAN_ROWS; r++) {
        const u32 word = p & 1 ? (((&w[r].x)[p >> 1]) >> 16) : (((&w[r].x)[p >> 1]) & 0xffffu);
        acc[2 * r] += (u64)word * v.x;
        acc[2 * r + 1] += (u64)word * v.y;
      }
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  warp_reduce8(acc, lane);
  // Lane l holds value x = ((l >> 4) & 1) 4 + ((l >> 3) & 1) 2 + ((l >> 2) & 1): row x / 2,
  // limb x & 1; a row's high limb sits four lanes above its low limb.
  const u64 hi = __shfl_down_sync(0xffffffffu, acc[0], 4);
  const int r = ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
  if ((lane & 7) == 0 && r < rows) out(r, (u128)acc[0] + ((u128)hi << 32));
}

// Tags of the columns of compact shards: the same sums over the words of the tag key that meet a column
// word's low half (its high half is zero). 64 columns a CTA share one staging of the key, where a warp a
// column read all of it each: 18.8 us a shard alone, part of one launch over all shards here.
template <int LOGN>
__global__ void __launch_bounds__(SCAN_WARPS * 32, 2) k_column_tags16(u32 gamma, const ShardDev* table, u32* mismatch) {
  constexpr int N = 1 << LOGN, M = N / 8;
  extern __shared__ __align__(16) uint4 scan_sm[];
  const ShardDev sh = table[blockIdx.y];
  if (!sh.cols16 || !sh.tag_key) return;
  const u32 j0 = blockIdx.x * SCAN_COLS + (threadIdx.x >> 5) * SCAN_ROWS;
  const int rows = j0 < gamma ? min(SCAN_ROWS, (int)(gamma - j0)) : 0;
  scan_columns16<LOGN>(
      scan_sm, sh.cols16 + (size_t)j0 * N, rows,
      [&](uint2* V) {
        for (int k = threadIdx.x; k < N; k += SCAN_WARPS * 32) {
          const u64 v = sh.tag_key[2 * k];
          V[(k & 7) * M + (k >> 3)] = make_uint2((u32)v, (u32)(v >> 32));
        }
      },
      [&](int r, u128 sum) { put_tag(sh, j0 + r, tag_residue(sum), mismatch); });
}

template <int LOGN>
__global__ void __launch_bounds__(SCAN_WARPS * 32, 2) k_scan(CrsDev c, const QueryDev* queries, const ShardDev* shards,
                                                          const u32* work, u32 chunks, u64* b_fold) {
  constexpr int N = 1 << LOGN, M = N / 8;
  extern __shared__ __align__(16) uint4 scan_sm[];
  u32 qi, chunk;
  if (work) {
    const u32 w = work[blockIdx.x];
    qi = w >> 12;
    chunk = w & 0xfff;
  } else {
    qi = blockIdx.x / chunks;
    chunk = blockIdx.x - qi * chunks;
  }
  // The respond launch that follows may start now: it takes the folds only at its end (scan_done).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const QueryDev qd = queries[qi];
  // b_rev in 32-bit limbs: every thread's loads of b issued first, beside the shard entry's.
  constexpr int PER = (N + SCAN_WARPS * 32 - 1) / (SCAN_WARPS * 32);
  u64 braw[PER];
#pragma unroll
  for (int j = 0; j < PER; j++) {
    const int k = threadIdx.x + j * SCAN_WARPS * 32;
    if (k < N) braw[j] = qd.b[k == 0 ? 0 : N - k];
  }
  const ShardDev sh = shards[qd.shard];
  const u32 gamma = qd.crs ? qd.crs->gamma : c.gamma;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const u32 j0 = chunk * SCAN_COLS + warp * SCAN_ROWS;
  const u64* b = qd.b;
  u64* fold_out = b_fold + qd.fold_off;
  const int rows = j0 < gamma ? min(SCAN_ROWS, (int)(gamma - j0)) : 0;

  if (sh.cols16) {
    scan_columns16<LOGN>(
        scan_sm, sh.cols16 + (size_t)j0 * N, rows,
        [&](uint2* V) {
#pragma unroll
          for (int j = 0; j < PER; j++) {
            const int k = threadIdx.x + j * SCAN_WARPS * 32;
            if (k >= N) break;
            const u64 bv = k == 0 ? reduce128(braw[j]) : negq(reduce128(braw[j]));
            V[(k & 7) * M + (k >> 3)] = make_uint2((u32)bv, (u32)(bv >> 32));
          }
        },
        [&](int r, u128 sum) { fold_out[j0 + r] = reduce128(sum); });
    return;
  }

#pragma unroll 1
  for (int r = 0; r < rows; r++) {
    const u32 j = j0 + r;
    const u64* col = sh.columns + (size_t)j * N;
    u128 flo = 0, fhi = 0;
#pragma unroll 4
    for (int k0 = lane * 2; k0 < N; k0 += 64) {
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(col + k0);
      const u64 r0 = k0 == 0 ? reduce128(b[0]) : negq(reduce128(b[N - k0]));
      const u64 r1 = negq(reduce128(b[N - k0 - 1]));
      const u128 p0 = (u128)w.x * r0, p1 = (u128)w.y * r1;
      flo += (u128)(u64)p0 + (u64)p1;
      fhi += (p0 >> 64) + (p1 >> 64);
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      flo += shfl_xor_u128(flo, m);
      fhi += shfl_xor_u128(fhi, m);
    }
    if (lane == 0) {
      // fold = fhi * 2^64 + flo (mod q)
      const u64 r64 = (u64)((((u128)1) << 64) % Q);
      const u64 hq = reduce128(fhi), lq = reduce128(flo);
      fold_out[j] = reduce128((u128)hq * r64 + lq);
    }
  }
}

// ServerResponse wire on the device (respond.rs:111-176, tight codec poly.rs:166-225):
// `tmpl` is the response with zero coefficients (header, lengths and trailer already in
// place); byte k of a packed region takes bits [8k, 8k+8) of the coefficients laid end to
// end at `bits` each, least significant first. One thread per output byte; a coefficient at
// or above the modulus sets status bit 1 of its response.
__global__ void k_wire(const u64* a, const u64* b, u32 n, u32 retained, u32 bits, u64 modulus, const uint8_t* tmpl,
                       u32 len, u32 a_off, u32 a_bytes, u32 b_off, u32 b_bytes, uint8_t* out, u32* status) {
  const u32 r = blockIdx.y;
  const u32 k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= len) return;
  u32 v = tmpl[k];
  const u64* c = nullptr;
  u32 count = 0, byte = 0;
  if (k >= a_off && k < a_off + a_bytes) {
    c = a + (size_t)r * n, count = n, byte = k - a_off;
  } else if (k >= b_off && k < b_off + b_bytes) {
    c = b + (size_t)r * n, count = retained, byte = k - b_off;
  }
  if (c) {
    const u64 bit = (u64)byte * 8;
    const u32 i0 = (u32)(bit / bits), sh = (u32)(bit - (u64)i0 * bits);
    u64 x = c[i0] >> sh;
    if (c[i0] >= modulus) atomicOr(status + r, 1u);
    if (sh + 8 > bits && i0 + 1 < count) x |= c[i0 + 1] << (bits - sh);
    v |= (u32)(x & 0xff);
  }
  out[(size_t)r * len + k] = (uint8_t)v;
}

// encode_database's column split (pir/encode_db.rs:74-168) for one shard: column j, row k
// holds bytes 2j and 2j+1 of entry k little-endian (one byte when the entry ends there,
// zero past it), rows past the last entry are zero. Writes the u64 words and their u16 copy.
//
// The entries are the rows of a transpose: a CTA takes ENC_ROWS entries by ENC_COLS columns through shared
// memory, reading along the entries and writing along the columns (a thread a word read its two bytes
// entry_size apart from its neighbours': 7.1 us a shard alone). Shard blockIdx.z of the launch holds entries
// n blockIdx.z onward of `rec`.
constexpr int ENC_ROWS = 64, ENC_COLS = 32;
__global__ void __launch_bounds__(256) k_encode_records(const uint8_t* rec, u64 total, u32 entry_size, u32 n, u32 gamma,
                                                        const ShardDev* table) {
  __shared__ uint16_t tile[ENC_COLS][ENC_ROWS + 2];
  const ShardDev sh = table[blockIdx.z];
  u64* cols = const_cast<u64*>(sh.columns);
  uint16_t* cols16 = const_cast<uint16_t*>(sh.cols16);
  const u64 first = (u64)blockIdx.z * n;
  const u32 entries = (u32)min((u64)n, total - first);
  rec += first * entry_size;
  const u32 k0 = blockIdx.y * ENC_ROWS, j0 = blockIdx.x * ENC_COLS;
  // One 16-byte load a thread where every entry starts on a 16-byte boundary (64 shards of 512-byte entries 92 -> 57 us),
  // two-byte loads where it starts on a two-byte one, single bytes otherwise.
  const bool wide = !(entry_size & 15) && !((size_t)rec & 15), pairs = !(entry_size & 1) && !((size_t)rec & 1);
  if (wide) {
    static_assert(ENC_ROWS * ENC_COLS / 8 == 256, "a load a thread");
    const u32 c = threadIdx.x % (ENC_COLS / 8), r = threadIdx.x / (ENC_COLS / 8), off = 2 * (j0 + 8 * c);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (k0 + r < entries && off < entry_size) v = *reinterpret_cast<const uint4*>(rec + (size_t)(k0 + r) * entry_size + off);
    const u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 8; q++) tile[8 * c + q][r] = (uint16_t)(w[q / 2] >> (16 * (q & 1)));
  }
  for (u32 i = threadIdx.x; i < ENC_ROWS * ENC_COLS && !wide; i += 256) {
    const u32 j = j0 + i % ENC_COLS, k = k0 + i / ENC_COLS, off = 2 * j;
    u32 v = 0;
    if (k < entries && off < entry_size) {
      const uint8_t* e = rec + (size_t)k * entry_size + off;
      if (pairs)
        v = *reinterpret_cast<const uint16_t*>(e);
      else
        v = off + 1 < entry_size ? (u32)e[0] | ((u32)e[1] << 8) : e[0];
    }
    tile[i % ENC_COLS][i / ENC_COLS] = (uint16_t)v;
  }
  __syncthreads();
  for (u32 i = threadIdx.x; i < ENC_ROWS * ENC_COLS / 2; i += 256) {
    const u32 j = j0 + i / (ENC_ROWS / 2), k = 2 * (i % (ENC_ROWS / 2));
    if (j >= gamma) continue;
    const u32 v = *reinterpret_cast<const u32*>(&tile[i / (ENC_ROWS / 2)][k]);
    const size_t at = (size_t)j * n + k0 + k;
    *reinterpret_cast<ulonglong2*>(cols + at) = make_ulonglong2(v & 0xffffu, v >> 16);
    *reinterpret_cast<u32*>(cols16 + at) = v;
  }
}

// Compact copy of a shard's columns: out[k] = w[k] when every word is below 2^16; any
// larger word sets *wide. Eight words per thread.
__global__ void k_compact16(const u64* cols, size_t groups, uint16_t* out, u32* wide) {
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= groups) return;
  const ulonglong2* src = reinterpret_cast<const ulonglong2*>(cols + 8 * g);
  u64 w[8];
  bool big = false;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const ulonglong2 v = src[k];
    w[2 * k] = v.x;
    w[2 * k + 1] = v.y;
    big |= (v.x | v.y) >> 16 != 0;
  }
  if (big) atomicOr(wide, 1u);
  uint4 o;
  o.x = (u32)w[0] | ((u32)w[1] << 16);
  o.y = (u32)w[2] | ((u32)w[3] << 16);
  o.z = (u32)w[4] | ((u32)w[5] << 16);
  o.w = (u32)w[6] | ((u32)w[7] << 16);
  reinterpret_cast<uint4*>(out)[g] = o;
}

// ------------------------------------------------------------------------------------
// Mod switch c' = floor((c q' + floor(q/2)) / q) mod q' (exact; q' < 2^62).
__device__ __forceinline__ u64 mod_switch_word(u64 cv, u64 qn) {
  const u128 x = (u128)cv * qn + (Q >> 1);
  u64 quo = (u64)(x >> 60);
  u128 r = x - (u128)quo * Q;
  while (r >= Q) {
    r -= Q;
    quo++;
  }
  return quo % qn;
}

// Rows X_0, X_1, X_2 (R-form, `stride` words apart, `dst_stride` in dst) of a 3-digit gadget key, folded for
// digits whose third transform is derived, D_2 = base^-2 (R - D_0 - base D_1):
//   sum_k X_k D_k = D_0 (X_0 - base^-2 X_2) + D_1 (X_1 - base^-1 X_2) + R base^-2 X_2.
// The folded rows are R-form too; a consumer then needs neither D_2 nor its reduction.
// Every read precedes every write, so src may equal dst.
__device__ __forceinline__ void fold_gadget3(u64 ld_inv_R, u64 ld_c0_R, u64 ld_c1_R, const u64* src, u64* dst,
                                             int stride, int dst_stride) {
  const u64 x0 = src[0], x1 = src[stride], x2 = src[2 * stride];
  const u64 f0 = addq(x0, mont(x2, ld_c0_R));
  const u64 f1 = addq(x1, mont(x2, ld_c1_R));
  const u64 f2 = mont(x2, ld_inv_R);
  dst[0] = f0;
  dst[dst_stride] = f1;
  dst[2 * dst_stride] = f2;
}

// The Galois keys ([key][digit][part][n], R-form NTT) folded by fold_gadget3, brought to standard form and laid out
// for the tree's threads: the pairs of a row's slots that thread u takes (2j, 2j + 1 of unit u) lie N/8 apart, so a
// warp's loads are contiguous (a thread's eight words in a row of their own took 16 wavefronts a load). The tree holds
// n^-1 times each node, so a digit's product is scaled by n^-1 and the node's own stays.
__global__ void k_fold_gadget_keys(CrsDev c, const u64* keys, u64* out, u32 count) {
  const u32 n = c.n;
  const u32 i = blockIdx.x * blockDim.x + threadIdx.x;  // (key, part, coefficient)
  if (i >= count * 2 * n) return;
  const u32 key = i / (2 * n), r = i - key * 2 * n, part = r / n, t = r - part * n;
  u64 x[3];
  fold_gadget3(c.ld_inv_R, c.ld_c0_R, c.ld_c1_R, keys + (size_t)key * 6 * n + r, x, (int)(2 * n), 1);
  u64* o = out + (size_t)key * 6 * n + (size_t)part * n + 2 * (((t & 7) >> 1) * (n / 8) + (t >> 3)) + (t & 1);
  o[0] = canon(mulw(x[0], c.s_ninv_rinv));
  o[2 * n] = canon(mulw(x[1], c.s_ninv_rinv));
  o[4 * n] = canon(mulw(x[2], c.s_rinv));
}

// The key rows of a mask or a seat as the recursion reads them, made once when the set or the seat is: per slot the
// rows of digits 0 and 1 side by side (2n words), then the row of the derived digit 2 (n words, exact gadget only).
// The recursion holds c_i = n^-1 R_i, so the inverse transform of a link needs no n^-1:
//   c_i = (n^-1 a)[tau] S + sum_k (n^-1 W_k)[tau] D_k,   sum_b += sum_k Y_k[tau] D_k,
// and with the exact gadget (rows folded as fold_gadget3 does), where R_{i+1} = n c_{i+1} takes the third digit's
// place, W_2 stays and Y_2 is scaled by n. A CTA a row, in one cluster: the fold reads the third row's transform from its
// CTA (13 us with the three transforms in one CTA). Folded by every
// respond CTA into its shared memory instead, the rows took 17,800 of the 123,000 cycles of a lone query of gamma 16.
template <int LOGN, int ROWS>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_key_rows(CrsDev c, const u64* in, u64* out, KeyScale f) {
  namespace cg = cooperative_groups;
  constexpr int N = 1 << LOGN, NT = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  Tw* tw = reinterpret_cast<Tw*>(sm);
  u64* x = sm + 2 * N;
  const int r = blockIdx.x;  // the CTA's row, and its rank in the cluster
  for (int k = threadIdx.x; k < N; k += NT) {
    tw[k] = c.tw[k];
    x[k] = reduce128(in[r * N + k]);
  }
  __syncthreads();
  {
    u64* const bufs[1] = {x};
    ntt_fwd_r4<LOGN, NT, 1>(bufs, tw);
  }
  cg::cluster_group cluster = cg::this_cluster();
  if constexpr (ROWS == 3) cluster.sync();
  const u64* third = ROWS == 3 ? cluster.map_shared_rank(x, 2) : x;
  const Tw fold = r ? f.fold1 : f.fold0;
  for (int k = threadIdx.x; k < N; k += NT) {
    if (r == 2) {
      out[2 * N + k] = canon(mulw(x[k], f.derived));
    } else {
      u64 y = mulw(x[k], f.digit);
      if constexpr (ROWS == 3) y += mulw(third[k], fold);
      out[2 * k + r] = canon(y);
    }
  }
  if constexpr (ROWS == 3) cluster.sync();  // the third row is read before its CTA ends
}

// A query's key rows in shared memory: W01 and Y01 the pairs of the mask and the seat, WY2 the third rows of both. The
// pointwise step gathers them with three 16-byte loads a slot.
struct KeyRows {
  ulonglong2 *W01, *Y01, *WY2;
};
__device__ __forceinline__ void stage_key_rows(const SetView& v, const u64* seat, const KeyRows& K, int n, int k, int to) {
  const u64* w = v.mask;
  const ulonglong2 w01 = reinterpret_cast<const ulonglong2*>(w)[k], y01 = reinterpret_cast<const ulonglong2*>(seat)[k];
  const bool exact = v.approx == 0;
  const ulonglong2 wy2 = make_ulonglong2(exact ? w[2 * n + k] : 0, exact ? seat[2 * n + k] : 0);
  K.W01[to] = w01;
  K.Y01[to] = y01;
  K.WY2[to] = wy2;
}
// The pointwise step of one slot at the gathered position tb: adds sum_k Y_k D_k to sb and returns
// c_i. d0, d1 at most 15q, cur at most 1+: sb takes at most 31 q^2 < 2^125 a call.
template <bool EXACT>
__device__ __forceinline__ u64 link_slot(Acc& sb, u64 d0, u64 d1, u64 cur, u64 s_R, const u64* a_ntt,
                                         const KeyRows& K, u32 tb) {
  const ulonglong2 w = K.W01[tb], y = K.Y01[tb];
  Acc r{0, 0, 0, 0};
  mac(r, a_ntt[tb], s_R);
  mac(r, d0, w.x);
  mac(sb, d0, y.x);
  mac(r, d1, w.y);
  mac(sb, d1, y.y);
  if constexpr (EXACT) {  // the rows are folded: c_{i+1} stands in for digit 2
    const ulonglong2 z = K.WY2[tb];
    mac(r, cur, z.x);
    mac(sb, cur, z.y);
  }
  return acc_fold(r);
}
// The links whose slot sums go without a fold: 4 x 2^125 and what is carried in stay below 2^128.
constexpr int SB_FOLD_LINKS = 4;

// The query's `a` in coefficient form: the ChaCha20 keystream of its seed as u64 words
// in order, each accepted by rand's gen_range(0..q) rule (math/poly.rs:657-671). Block b
// of the stream yields words 8b..8b+7; a rejected word (probability ~2^-46) shifts every
// later coefficient, and the walk is then redone word by word. Ends with a barrier.
template <int N, int NT>
__device__ __forceinline__ void expand_a(const QueryDev& qd, u64* a, u32* status, u32 qi, int force_serial) {
  const int tid = threadIdx.x;
  bool rejected = false;
  if (qd.a) {
    for (int k = tid; k < N; k += NT) a[k] = reduce128(qd.a[k]);
  } else if (tid < N / 8) {
    u32 blk[16], key[8];
#pragma unroll
    for (int k = 0; k < 8; k++) key[k] = qd.seed[k];
    chacha20_block(key, (u64)tid, 0, blk);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const u64 v = (u64)blk[2 * k] | ((u64)blk[2 * k + 1] << 32);
      if (v * Q > RANGE_ZONE) rejected = true;
      a[tid * 8 + k] = mulhi(v, Q);
    }
  }
  if (__syncthreads_or(rejected || (force_serial && !qd.a))) {
    if (tid == 0) {
      u32 blk[16], key[8];
      for (int k = 0; k < 8; k++) key[k] = qd.seed[k];
      u64 have = ~0ULL, cand = 0;
      int filled = 0;
      const u64 limit = (u64)N + 65536;
      while (filled < N && cand < limit) {
        const u64 bi = cand >> 3;
        if (bi != have) {
          chacha20_block(key, bi, 0, blk);
          have = bi;
        }
        const int k = (int)(cand & 7);
        const u64 v = (u64)blk[2 * k] | ((u64)blk[2 * k + 1] << 32);
        if (v * Q <= RANGE_ZONE) a[filled++] = mulhi(v, Q);
        cand++;
      }
      if (filled < N) {
        atomicOr(status + qi, (u32)DEV_EXPAND_EXHAUSTED);
        for (; filled < N; filled++) a[filled] = 0;
      }
    }
    __syncthreads();
  }
}

// Waits for the launch's scan, which runs beside the recursion (programmatic launch): called before the first use of
// a b fold.
__device__ __forceinline__ void scan_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Refuses a query on a stale shard. The respond kernel itself checks, on the table entry that it takes the store from and
// before its first use: its scan runs beside it, and a store rebuilt between the two reads would pass for a good one.
__device__ __forceinline__ void refuse_stale(const ShardDev& sh, u32* status, u32 qi) {
  if (sh.stale) atomicOr(status + qi, (u32)DEV_TAG_MISMATCH);
}

// Coefficients of the response from the unscaled inverse transforms of c_0 = n^-1 R_0 (a) and of
// the online sum (b).
__device__ __forceinline__ u64 finish_a(u64 x, u64 ms) {
  const u64 v = canon(x);
  return ms ? mod_switch_word(v, ms) : v;
}
__device__ __forceinline__ u64 finish_b(const CrsDev& c, u64 x, u32 t, u32 gamma, const u64* fold, u64 ms) {
  u64 v = canon(mulw(x, c.ninv));
  if (t < gamma) v = addq(v, fold[t]);
  return ms ? mod_switch_word(v, ms) : v;
}

// The digits 0 and 1 of a canonical coefficient: base 2^20, of the coefficient itself (exact) or of
// its rounding to a multiple of 2^20 with the lowest digit dropped (the top carry is kept).
template <bool EXACT>
__device__ __forceinline__ void split_digits(u64 r, u32& g0, u32& g1) {
  constexpr u32 DMASK = (1u << 20) - 1;
  if constexpr (EXACT) {
    g0 = (u32)r & DMASK;
    g1 = (u32)(r >> 20) & DMASK;
  } else {
    const u64 rr = (r + (1ULL << 19)) >> 20;
    g0 = (u32)rr & DMASK;
    g1 = (u32)(rr >> 20);
  }
}

constexpr int FWD_FREE = 9;  // a radix-4 unit whose words are at most this needs no reduction: 9 + 6 < 16

// ------------------------------------------------------------------------------------
// Radix-8 transforms of one CTA of N/8 threads (the one-CTA respond kernel): three stages a
// shared-memory round trip on units of eight words a thread. Against radix-4 passes on N/4 threads
// a link takes 6 barriers instead of 10 and half the shared-memory wavefronts (2.26 M -> 1.14 M a query at
// gamma 256), and each phase between barriers is long enough to hide its loads: 7.14 -> 6.79 ms for 509
// queries. What bounds it now is the two warps a sub-partition that its shared memory leaves room for:
// the heavy multiply pipe is busy 70% of cycles, the warps' fixed-latency waits take the rest.
//
// Layouts, free of bank conflicts in every pass of the 2048 ring:
//   sw8    words of the transform buffers: bits 4-5 of the index XORed into bits 1-2 spread the
//          16-byte accesses of contiguous units, bit 6 into bit 3 those of the stride-8 passes;
//   tw8    ladder entries: the levels N/4 and N/2, used only by the passes on contiguous units, hold
//          the entries that a unit takes N/8 apart, so a warp's loads are contiguous;
//   slot8  gathered operands (a_ntt, the key rows): slot t at (t & 7) N/8 + (t >> 3). The slots
//          8 l + k of a warp's lanes l go to slots whose t >> 3 differ modulo any power of two that
//          theirs do (an odd affine map of the bit-reversed index), so a gather hits distinct banks.
__device__ __forceinline__ int sw8(int e) { return e ^ (((e >> 4) & 3) << 1) ^ (((e >> 6) & 1) << 3); }
template <int LOGN>
__device__ __forceinline__ int tw8(int m) {
  constexpr int N = 1 << LOGN, E = N / 8;
  if (m >= N / 2) return N / 2 + (m & 3) * E + ((m - N / 2) >> 2);
  if (m >= N / 4) return N / 4 + (m & 1) * E + ((m - N / 4) >> 1);
  return m;
}
template <int LOGN>
__device__ __forceinline__ int slot8(int t) {
  return ((t & 7) << (LOGN - 3)) | (t >> 3);
}

// Three forward stages; out <= in + 9. RED brings the words that are not multiplied first down to 1.
template <bool RED>
__device__ __forceinline__ void fwd_unit8(u64 (&x)[8], const Tw& w0, const Tw (&w1)[2], const Tw (&w2)[4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (RED) x[k] = red60(x[k]);
    bf_fwd(x[k], x[k + 4], w0);
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    bf_fwd(x[k], x[k + 2], w1[0]);
    bf_fwd(x[k + 4], x[k + 6], w1[1]);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) bf_fwd(x[2 * k], x[2 * k + 1], w2[k]);
}
constexpr int FWD_FREE8 = 6;  // 6 + 9 < 16

// Three inverse stages on words up to 2+; out at most 2+. The first word's sum after two stages (8+)
// is reduced before it meets its equal, and the four sums at the end.
__device__ __forceinline__ void inv_unit8(u64 (&x)[8], const Tw (&f0)[4], const Tw (&f1)[2], const Tw& f2) {
#pragma unroll
  for (int k = 0; k < 4; k++) bf_inv<3>(x[2 * k], x[2 * k + 1], f0[k]);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    bf_inv<5>(x[4 * k], x[4 * k + 2], f1[k]);
    bf_inv<3>(x[4 * k + 1], x[4 * k + 3], f1[k]);
  }
  x[0] = red60(x[0]);
  bf_inv<2>(x[0], x[4], f2);
  bf_inv<5>(x[1], x[5], f2);
  bf_inv<3>(x[2], x[6], f2);
  bf_inv<3>(x[3], x[7], f2);
#pragma unroll
  for (int k = 0; k < 4; k++) x[k] = red60(x[k]);
}

// Stages a middle pass takes with `rem` left: three, but two and two of four, and two of two.
__host__ __device__ constexpr int pass_stages(int rem) { return rem == 4 || rem == 2 ? 2 : 3; }

// Inverse stages S .. logn-3 of NB buffers N words apart, words up to 2+ in and out. Each pass ends with
// a barrier.
template <int LOGN, int NB, int S = 3>
__device__ __forceinline__ void inv_middle8(u64* X, const Tw* tw) {
  constexpr int N = 1 << LOGN, NT = N / 8;
  if constexpr (S < LOGN - 2) {
    constexpr int K = pass_stages(LOGN - 2 - S), t = 1 << S, M = N >> (S + 1);
    if constexpr (K == 3) {
      const int u = threadIdx.x, B = u >> S, o = u & (t - 1), e0 = B * 8 * t + o;
      Tw f0[4], f1[2];
#pragma unroll
      for (int j = 0; j < 4; j++) f0[j] = tw[2 * M - 1 - 4 * B - j];
#pragma unroll
      for (int j = 0; j < 2; j++) f1[j] = tw[M - 1 - 2 * B - j];
      const Tw f2 = tw[M / 2 - 1 - B];
#pragma unroll
      for (int n = 0; n < NB; n++) {
        u64 x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = X[n * N + sw8(e0 + k * t)];
        inv_unit8(x, f0, f1, f2);
#pragma unroll
        for (int k = 0; k < 8; k++) X[n * N + sw8(e0 + k * t)] = x[k];
      }
    } else {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int u = threadIdx.x + r * NT, B = u >> S, o = u & (t - 1), e0 = B * 4 * t + o;
#pragma unroll
        for (int n = 0; n < NB; n++) {
          u64 x[4];
#pragma unroll
          for (int k = 0; k < 4; k++) x[k] = X[n * N + sw8(e0 + k * t)];
          inv_unit(x[0], x[1], x[2], x[3], tw[2 * M - 1 - 2 * B], tw[2 * M - 2 - 2 * B], tw[M - 1 - B]);
#pragma unroll
          for (int k = 0; k < 4; k++) X[n * N + sw8(e0 + k * t)] = x[k];
        }
      }
    }
    __syncthreads();
    inv_middle8<LOGN, NB, S + K>(X, tw);
  }
}

// Forward stages S .. logn-4 of NB buffers N words apart, words up to BIN in and fwd_bound8 out. Each pass
// ends with a barrier.
__host__ __device__ constexpr int fwd_bound8(int logn, int s, int b) {
  for (; s < logn - 3; s += pass_stages(logn - 3 - s)) {
    const int k = pass_stages(logn - 3 - s);
    b = (b > 15 - 3 * k ? 1 : b) + 3 * k;
  }
  return b;
}
template <int LOGN, int NB, int BIN, int S = 2>
__device__ __forceinline__ void fwd_middle8(u64* D, const Tw* tw) {
  constexpr int N = 1 << LOGN, NT = N / 8;
  if constexpr (S < LOGN - 3) {
    constexpr int K = pass_stages(LOGN - 3 - S), m = 1 << S, h = N >> (S + K);
    constexpr bool RED = BIN > 15 - 3 * K;
    if constexpr (K == 3) {
      const int u = threadIdx.x, i = u / h, o = u % h, e0 = i * 8 * h + o;
      const Tw w0 = tw[m + i];
      Tw w1[2], w2[4];
#pragma unroll
      for (int j = 0; j < 2; j++) w1[j] = tw[2 * m + 2 * i + j];
#pragma unroll
      for (int j = 0; j < 4; j++) w2[j] = tw[4 * m + 4 * i + j];
#pragma unroll
      for (int n = 0; n < NB; n++) {
        u64 x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = D[n * N + sw8(e0 + k * h)];
        fwd_unit8<RED>(x, w0, w1, w2);
#pragma unroll
        for (int k = 0; k < 8; k++) D[n * N + sw8(e0 + k * h)] = x[k];
      }
    } else {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int u = threadIdx.x + r * NT, i = u / h, o = u % h, e0 = i * 4 * h + o;
#pragma unroll
        for (int n = 0; n < NB; n++) {
          u64 x[4];
#pragma unroll
          for (int k = 0; k < 4; k++) x[k] = D[n * N + sw8(e0 + k * h)];
          fwd_unit<RED>(x[0], x[1], x[2], x[3], tw[m + i], tw[2 * m + 2 * i], tw[2 * m + 2 * i + 1]);
#pragma unroll
          for (int k = 0; k < 4; k++) D[n * N + sw8(e0 + k * h)] = x[k];
        }
      }
    }
    __syncthreads();
    fwd_middle8<LOGN, NB, (RED ? 1 : BIN) + 3 * K, S + K>(D, tw);
  }
}

// The first three inverse stages of thread tid's unit (slots 8 tid .. 8 tid + 7, words up to 2+), from
// registers to X.
template <int LOGN>
__device__ __forceinline__ void inv_first8(u64 (&x)[8], u64* X, const Tw* tw) {
  constexpr int N = 1 << LOGN, E = N / 8;
  const int tid = threadIdx.x, r = E - 1 - tid;  // the mirrored unit
  Tw f0[4], f1[2];
#pragma unroll
  for (int j = 0; j < 4; j++) f0[j] = tw[N / 2 + (3 - j) * E + r];
#pragma unroll
  for (int j = 0; j < 2; j++) f1[j] = tw[N / 4 + (1 - j) * E + r];
  inv_unit8(x, f0, f1, tw[E + r]);
#pragma unroll
  for (int k = 0; k < 8; k += 2)
    *reinterpret_cast<ulonglong2*>(X + sw8(8 * tid + k)) = make_ulonglong2(x[k], x[k + 1]);
}

// The last three forward stages of thread tid's unit of NB buffers, to registers: at most 15.
template <int LOGN, int NB, int BIN>
__device__ __forceinline__ void fwd_last8(u64 (&x)[NB][8], const u64* D, const Tw* tw) {
  constexpr int N = 1 << LOGN, E = N / 8;
  constexpr bool RED = BIN > FWD_FREE8;
  const int tid = threadIdx.x;
  const Tw w0 = tw[E + tid];
  Tw w1[2], w2[4];
#pragma unroll
  for (int j = 0; j < 2; j++) w1[j] = tw[N / 4 + j * E + tid];
#pragma unroll
  for (int j = 0; j < 4; j++) w2[j] = tw[N / 2 + j * E + tid];
#pragma unroll
  for (int n = 0; n < NB; n++) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(D + n * N + sw8(8 * tid + k));
      x[n][k] = v.x;
      x[n][k + 1] = v.y;
    }
    fwd_unit8<RED>(x[n], w0, w1, w2);
  }
}

// One link's transforms: thread tid holds the NTT-domain words cur of its unit (at most 1+, scaled by
// n^-1) and gets the transforms of digits 0 and 1 of their inverse transform at the same slots, at most
// 15. The inverse's last two stages, the digit split and the forward's first two are one radix-4 pass
// over the words b + k N/4. D: 2N words; the inverse runs in the first N, which the pass rewrites in
// place as digit 0. No thread touches another's unit after the last barrier, so the next link may
// follow without one.
template <int LOGN, bool EXACT>
__device__ __forceinline__ void link_transforms8(const u64 (&cur)[8], u64 (&d)[2][8], u64* D, const Tw* tw) {
  constexpr int N = 1 << LOGN, NT = N / 8, P = N / 4;
  {
    u64 x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = cur[k];
    inv_first8<LOGN>(x, D, tw);
  }
  __syncthreads();
  inv_middle8<LOGN, 1>(D, tw);
  const Tw w1 = tw[1], w2 = tw[2], w3 = tw[3];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int b = threadIdx.x + j * NT;
    u64 x[4];
    int at[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = D[at[k] = sw8(b + k * P)];
    bf_inv<3>(x[0], x[1], w3);
    bf_inv<3>(x[2], x[3], w2);
    u32 g[2][4];
    split_digits<EXACT>(canon(x[0] + x[2]), g[0][0], g[1][0]);
    split_digits<EXACT>(canon(x[1] + x[3]), g[0][1], g[1][1]);
    split_digits<EXACT>(canon(mulw(x[2] - x[0] + 5 * Q, w1)), g[0][2], g[1][2]);
    split_digits<EXACT>(canon(mulw(x[3] - x[1] + 3 * Q, w1)), g[0][3], g[1][3]);
#pragma unroll
    for (int n = 0; n < 2; n++) {
      const u64 t2 = mulw_digit(g[n][2], w1), t3 = mulw_digit(g[n][3], w1);
      u64 y0 = g[n][0] + t2, y2 = g[n][0] + 3 * Q - t2, y1 = g[n][1] + t3, y3 = g[n][1] + 3 * Q - t3;
      bf_fwd(y0, y1, w2);
      bf_fwd(y2, y3, w3);
      D[n * N + at[0]] = y0;
      D[n * N + at[1]] = y1;
      D[n * N + at[2]] = y2;
      D[n * N + at[3]] = y3;
    }
  }
  __syncthreads();
  fwd_middle8<LOGN, 2, 6>(D, tw);
  fwd_last8<LOGN, 2, fwd_bound8(LOGN, 2, 6)>(d, D, tw);
}

// scale NTT(src), canonical, at the thread's slots (src: N coefficients in plain order). D: N words of scratch
// other than src.
template <int LOGN>
__device__ __forceinline__ void transform_slots8(const u64* src, u64* D, const Tw* tw, const Tw& scale, u64 (&out)[8]) {
  constexpr int N = 1 << LOGN, NT = N / 8, P = N / 4;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int b = threadIdx.x + j * NT;
    u64 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = src[b + k * P];
    fwd_unit<false>(x[0], x[1], x[2], x[3], tw[1], tw[2], tw[3]);
#pragma unroll
    for (int k = 0; k < 4; k++) D[sw8(b + k * P)] = x[k];
  }
  __syncthreads();
  fwd_middle8<LOGN, 1, 7>(D, tw);
  u64 x[1][8];
  fwd_last8<LOGN, 1, fwd_bound8(LOGN, 2, 7)>(x, D, tw);
#pragma unroll
  for (int k = 0; k < 8; k++) out[k] = canon(mulw(x[0][k], scale));
}

// The column transforms of a store build, several shards a launch (blockIdx.y): H row j is the transform of
// column j, left lazy (at most 15, the fold takes any word). A CTA stages the ladder once for
// STORE_ROWS columns; compact columns are read from their u16 copy, and their first stage takes the
// 32-bit product.
constexpr int STORE_ROWS = 4;
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8, 4) k_store_ntt(CrsDev c, ShardArg shards, u64* H) {
  constexpr int N = 1 << LOGN, NT = N / 8, P = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  Tw* tw = reinterpret_cast<Tw*>(sm);
  u64* D = sm + 2 * N;
  const ShardDev sh = shard_of(shards);
  for (int k = threadIdx.x; k < N; k += NT) tw[tw8<LOGN>(k)] = c.tw[k];
  __syncthreads();
  H += (size_t)blockIdx.y * c.gamma * N;
  const u32 end = min(c.gamma, (blockIdx.x + 1) * STORE_ROWS);
  u32 next[2][4] = {};  // the next compact column's words
  auto fetch = [&](u32 j) {
    if (!sh.cols16 || j >= end) return;
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int k = 0; k < 4; k++) next[r][k] = sh.cols16[(size_t)j * N + threadIdx.x + r * NT + k * P];
  };
  fetch(blockIdx.x * STORE_ROWS);
#pragma unroll 1
  for (u32 j = blockIdx.x * STORE_ROWS; j < end; j++) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int b = threadIdx.x + r * NT;
      u64 x[4];
      if (sh.cols16) {
        const u32(&w)[4] = next[r];
        const u64 t2 = mulw_digit(w[2], tw[1]), t3 = mulw_digit(w[3], tw[1]);
        x[0] = w[0] + t2;
        x[1] = w[1] + t3;
        x[2] = w[0] + 3 * Q - t2;
        x[3] = w[1] + 3 * Q - t3;
        bf_fwd(x[0], x[1], tw[2]);
        bf_fwd(x[2], x[3], tw[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = red60(sh.columns[(size_t)j * N + b + k * P]);
        fwd_unit<false>(x[0], x[1], x[2], x[3], tw[1], tw[2], tw[3]);
      }
#pragma unroll
      for (int k = 0; k < 4; k++) D[sw8(b + k * P)] = x[k];
    }
    fetch(j + 1);  // while this one is transformed
    __syncthreads();
    fwd_middle8<LOGN, 1, 7>(D, tw);
    u64 x[1][8];
    fwd_last8<LOGN, 1, fwd_bound8(LOGN, 2, 7)>(x, D, tw);
    ulonglong2* o = reinterpret_cast<ulonglong2*>(H + (size_t)j * N + 8 * threadIdx.x);
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = make_ulonglong2(x[0][2 * k], x[0][2 * k + 1]);
    __syncthreads();  // D is rewritten by the next column
  }
}

// The recursion's links gamma - 2 .. 0 on thread tid's slots (sums: the store's row 0 at its first slot).
template <int LOGN, bool EXACT>
__device__ __forceinline__ void respond_links8(u64 (&cur)[8], Acc (&sb)[8], const u32 (&et)[8], u32 gamma,
                                               const u32* gpow, const u64* sums, u64* D, const u64* a_ntt,
                                               const Tw* tw, const KeyRows& K, const uint16_t* s_tab) {
  constexpr int N = 1 << LOGN;
  constexpr u32 M2N = 2 * N - 1;
#pragma unroll 1
  for (int i = (int)gamma - 2; i >= 0; i--) {
    const ulonglong2* Srow = reinterpret_cast<const ulonglong2*>(sums + (size_t)i * N);
    ulonglong2 sv[4];
#pragma unroll
    for (int k = 0; k < 4; k++) sv[k] = Srow[k];
    const u32 gp = gpow[i];
    u64 d[2][8];
    link_transforms8<LOGN, EXACT>(cur, d, D, tw);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const u32 tb = s_tab[((gp * et[k]) & M2N) >> 1];
      cur[k] = link_slot<EXACT>(sb[k], d[0][k], d[1][k], cur[k], k & 1 ? sv[k / 2].y : sv[k / 2].x, a_ntt, K, tb);
    }
    if (i % SB_FOLD_LINKS == 0) {
#pragma unroll
      for (int k = 0; k < 8; k++) sb[k] = acc_from(acc_fold(sb[k]));
    }
  }
}

// One CTA per query (batches that fill the GPU). Thread u owns slots 8u..8u+7 of every
// NTT-domain vector (one transform unit). Each link of the recursion (i from gamma-2 down
// to 0) holds n^-1 R_{i+1} in NTT form (`cur`, in registers):
//   r = INTT(R_{i+1});  d_k = base-2^20 digits of r (rounded, top carry kept, when the
//   lowest digit is dropped);  D_k = NTT(d_k);
//   sum_b += sum_k Y_k[tau_i(t)] D_k[t];
//   R_i[t] = a_ntt[tau_i(t)] S_i[t] + sum_k W_k[tau_i(t)] D_k[t]
// with tau_i the slot permutation of the automorphism X -> X^(g^i), S the packing store,
// W the mask rows and Y the seat. Digits 0 and 1 are transformed; with the exact gadget
// digit 2's transform is D_2 = base^-2 (R_{i+1} - D_0 - base D_1) (inspiring2.rs:1094-1161),
// a fixed linear combination, so the key rows hold it folded (k_key_rows) and
// R_{i+1} takes digit 2's place in the sums.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8, 1)
    k_respond(CrsDev c, const QueryDev* queries, const ShardDev* shards, const u64* b_fold, u64* a_out, u64* b_out,
              u32* status, int force_serial) {
  constexpr int N = 1 << LOGN, NT = N / 8, P = N / 4;
  constexpr u32 M2N = 2 * N - 1;
  extern __shared__ __align__(16) u64 sm[];
  u64* D = sm;  // 2N: the inverse in progress in the first N, then digits 0 and 1
  u64* a_ntt = D + 2 * N;
  Tw* tw = reinterpret_cast<Tw*>(a_ntt + N);
  // Room for three key rows whatever the query's gadget, so queries of different sets
  // share a launch.
  ulonglong2* rows = reinterpret_cast<ulonglong2*>(tw + N);
  const KeyRows K{rows, rows + N, rows + 2 * N};
  uint16_t* s_tab = reinterpret_cast<uint16_t*>(rows + 3 * N);  // position of the slot of exponent 2e + 1

  // The launch of a batch's tail may follow as SMs come free (it waits for this one's end at its own: scan_done).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x;
  const QueryDev qd = queries[blockIdx.x];
  const u32 qi = qd.row;  // output and status row
  const ShardDev sh = shards[qd.shard];
  const SetView ps = set_view(c, qd.crs);
  const u32 gamma = ps.gamma;
  const bool exact = ps.approx == 0;
  const int l0 = 8 * tid;
  if (tid == 0) refuse_stale(sh, status, qi);

#pragma unroll 4
  for (int k = tid; k < N; k += NT) stage_key_rows(ps, qd.seat, K, N, k, slot8<LOGN>(k));
#pragma unroll 8
  for (int k = tid; k < N; k += NT) {
    tw[tw8<LOGN>(k)] = c.tw[k];
    s_tab[k] = (uint16_t)slot8<LOGN>(c.exp_slot[k]);
  }
  expand_a<N, NT>(qd, D + N, status, qi, force_serial);  // ends with a barrier
  {
    // n^-1 2^-64 NTT(a): the factor that takes an R-form store word to c_i's scale.
    u64 x[8];
    transform_slots8<LOGN>(D + N, D, tw, c.s_ninv_rinv, x);
#pragma unroll
    for (int k = 0; k < 8; k++) a_ntt[k * NT + tid] = x[k];
    __syncthreads();
  }

  u64 cur[8];
  Acc sb[8];
  u32 et[8];
  {
    const u32 gp = ps.gpow[gamma - 1];
    const u64* Srow = sh.sums_R + (size_t)(gamma - 1) * N + l0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      et[k] = c.slot_exp[l0 + k];
      cur[k] = mulq(a_ntt[s_tab[((gp * et[k]) & M2N) >> 1]], Srow[k]);
      sb[k] = Acc{0, 0, 0, 0};
    }
  }
  if (exact)
    respond_links8<LOGN, true>(cur, sb, et, gamma, ps.gpow, sh.sums_R + l0, D, a_ntt, tw, K, s_tab);
  else
    respond_links8<LOGN, false>(cur, sb, et, gamma, ps.gpow, sh.sums_R + l0, D, a_ntt, tw, K, s_tab);
  // Final inverse transforms of c_0 (to a) and of the online sum (to b), in the two halves of D.
  {
    u64 x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = acc_fold(sb[k]);
    inv_first8<LOGN>(cur, D, tw);
    inv_first8<LOGN>(x, D + N, tw);
  }
  __syncthreads();
  inv_middle8<LOGN, 2>(D, tw);
  scan_done();
  const Tw w1 = tw[1], w2 = tw[2], w3 = tw[3];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int b = tid + j * NT;
#pragma unroll
    for (int n = 0; n < 2; n++) {
      u64 x[4];
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = D[n * N + sw8(b + k * P)];
      inv_unit(x[0], x[1], x[2], x[3], w3, w2, w1);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int t = b + k * P;
        if (n == 0)
          a_out[(size_t)qi * N + t] = finish_a(x[k], qd.ms);
        else
          b_out[(size_t)qi * N + t] = finish_b(c, x[k], t, gamma, b_fold + qd.fold_off, qd.ms);
      }
    }
  }
}

// ------------------------------------------------------------------------------------
// A cluster of R = 2 or 4 CTAs per query, for batches that leave SMs idle with one CTA each: a query's
// recursion spread over R SMs, where the time of a link is its chain of dependent steps.
//
// CTA r owns part r, words [r P, (r+1) P), P = N/R, of every NTT-domain vector, two words a thread. The
// inverse (Gentleman-Sande, from t = 1 upward) stays inside a part for its first log P stages and the forward
// (Cooley-Tukey, downward) for its last log P; the log R stages between them mix word e of every part.
// Per link:
//   1. local inverse: stage 0 on the thread's own pair, then radix-4 units through shared memory on half the
//      threads (one unit a thread, its two stages in registers). Units on bits 1-6 stay within the 128
//      words of a warp, so a warp barrier between them is enough; bits 7 and up take a CTA barrier. (One
//      butterfly a thread with lane exchanges keeps every thread busy, but its selects cost the ALU
//      port half as much again as the products: 1,300 cycles for nine stages.)
//   2. each word goes to the CTA that crosses its e (CTA e / (P/R)), by an asynchronous store to its shared
//      memory that counts on an mbarrier there.
//   3. the cross: the inverse's last log R stages, the digit split, the forward's first log R stages, for
//      P/R words a CTA and not all P (each CTA computing every cross and keeping its own part took 2,160
//      cycles); the digits' words go back to their owners the same way.
//   4. local forward of both digits, the inverse's passes backwards with a unit of one digit a thread, ending with
//      both digits of the thread's own pair.
//   5. the pointwise step. The online sum is off the chain, so its products run while the cross words travel, and
//      the products of a, S and c_{i+1} while the digits do: 64 queries of gamma 256 1.27 -> 1.16 ms, 33 of gamma
//      1024 2.97 -> 2.84 ms.
// Setup: each CTA transforms its part of a and sends the slots to every CTA (each transforming all of it, and staging
// one load a thread at a time: 30,700 -> 14,800 cycles, a lone query of gamma 16 122 -> 112 us with the end below).
// A link of four CTAs now takes 5,000 cycles: inverse 1,600, its exchange 610, cross 820, the digits' 220, forward
// 1,180, pointwise 570. Two CTAs an SM (the seat's rows from L2, half the shared memory) ran 64 queries no faster
// than clusters of two: both share the multiply pipe.
// The data's own arrivals order the reuse of the exchange buffers. A CTA sends a link's cross words after its forward of
// the link before, which took digits from every peer, and a peer sends those after reading its cross words; it sends
// digits after taking cross words from every peer, and a peer's threads send those after reading their
// digits of the link before. X is a CTA's own: between two links the forward's last barrier orders its reuse, between
// the two final transforms a barrier of its own.
template <int LOGN, int R>
struct Part {
  static constexpr int N = 1 << LOGN, LR = R == 4 ? 2 : 1, LP = LOGN - LR, P = 1 << LP, NT = P / 2;
  static constexpr int C = P / R;  // words whose cross a CTA computes
  // The part's words in shared memory: every pass's accesses are free of bank conflicts.
  static __device__ __forceinline__ int sw(int e) { return e ^ (((e >> 4) & 3) << 1) ^ (((e >> 5) & 1) << 3); }
  // First word of unit u of a pass on `n` index bits from bit b (word k of the unit: + k 2^b).
  static __device__ __forceinline__ int unit(int u, int b, int n) { return ((u >> b) << (b + n)) | (u & ((1 << b) - 1)); }
  static __host__ __device__ constexpr int bits(int b) { return b + 1 < LP ? 2 : 1; }  // of the pass from bit b (odd)
};

// A part's ladders: level m' (entries m' + i, i < m') holds the ring's level m' R at the entries of the part's blocks
// for the forward, at those of the mirrored part's for the inverse.
template <int R>
__device__ __forceinline__ int part_ladder(int k, int part) {
  const int m = 1 << (31 - __clz(k));
  return m * (R + part) + (k - m);
}

// Local inverse stages from bit B up, on the part's words X (2+ in and out); put(e, word) takes the last
// pass's words instead of X. tw: the mirrored part's ladder.
template <int LOGN, int R, int B, class Put>
__device__ __forceinline__ void part_inverse(u64* X, const Tw* tw, Put put) {
  using G = Part<LOGN, R>;
  if constexpr (B < G::LP) {
    constexpr int n = G::bits(B), t = 1 << B, M = G::P >> (B + 1);
    constexpr bool last = B + n == G::LP;
    if ((int)threadIdx.x < (G::P >> n)) {
      const int e = G::unit(threadIdx.x, B, n), i = e >> (B + 1);
      u64 x[1 << n];
#pragma unroll
      for (int k = 0; k < 1 << n; k++) x[k] = X[G::sw(e + k * t)];
      if constexpr (n == 2) {
        inv_unit(x[0], x[1], x[2], x[3], tw[2 * M - 1 - i], tw[2 * M - 2 - i], tw[M - 1 - (i >> 1)]);
      } else {
        bf_inv<3>(x[0], x[1], tw[2 * M - 1 - i]);
        x[0] = red60(x[0]);
      }
#pragma unroll
      for (int k = 0; k < 1 << n; k++) {
        if constexpr (last)
          put(e + k * t, k, x[k]);
        else
          X[G::sw(e + k * t)] = x[k];
      }
    }
    if constexpr (!last) {
      if constexpr (B + n >= 7)
        __syncthreads();
      else
        __syncwarp();
    }
    part_inverse<LOGN, R, B + n>(X, tw, put);
  }
}

// Local forward stages from the pass at bit B down to bit 1, both digits in place (D[0..P), D[P..2P)), words
// up to W in and part_bound out. tw: the part's ladder. Ends with a CTA barrier.
__host__ __device__ constexpr int part_bound(int lp, int b, int w) {
  for (; b >= 1; b -= 2) w = b + 1 < lp ? (w > FWD_FREE ? 1 : w) + 6 : (w > 12 ? 1 : w) + 3;
  return w;
}
template <int LOGN, int R, int B, int W>
__device__ __forceinline__ void part_forward(u64* D, const Tw* tw) {
  using G = Part<LOGN, R>;
  if constexpr (B >= 1) {
    constexpr int n = G::bits(B), t = 1 << B, m = G::P >> (B + n);
    constexpr bool RED = n == 2 ? W > FWD_FREE : W > 12;
    if constexpr (n == 2) {  // a unit of one digit a thread
      const int u = threadIdx.x & (G::P / 4 - 1);
      u64* x = D + ((int)threadIdx.x < G::P / 4 ? 0 : G::P);
      const int e = G::unit(u, B, 2), i = e >> (B + 2);
      const int i0 = G::sw(e), i1 = G::sw(e + t), i2 = G::sw(e + 2 * t), i3 = G::sw(e + 3 * t);
      u64 a0 = x[i0], a1 = x[i1], a2 = x[i2], a3 = x[i3];
      fwd_unit<RED>(a0, a1, a2, a3, tw[m + i], tw[2 * m + 2 * i], tw[2 * m + 2 * i + 1]);
      x[i0] = a0;
      x[i1] = a1;
      x[i2] = a2;
      x[i3] = a3;
    } else {  // a pair of each digit a thread
      const int e = G::unit(threadIdx.x, B, 1), i0 = G::sw(e), i1 = G::sw(e + t);
      const Tw w = tw[m + (e >> (B + 1))];
#pragma unroll
      for (int d = 0; d < 2; d++) {
        u64* x = D + d * G::P;
        u64 a = x[i0], c = x[i1];
        if (RED) a = red60(a);
        bf_fwd(a, c, w);
        x[i0] = a;
        x[i1] = c;
      }
    }
    if constexpr (B >= 7 || B == 1)
      __syncthreads();
    else
      __syncwarp();
    part_forward<LOGN, R, B - 2, (RED ? 1 : W) + 3 * n>(D, tw);
  }
}

// The inverse's last log R stages on word e of the R parts (words up to 2+): canonical coefficients.
template <int R>
__device__ __forceinline__ void cross_inverse(const u64 (&x)[R], u64 (&cf)[R], const Tw& w1, const Tw& w2, const Tw& w3) {
  if constexpr (R == 2) {
    cf[0] = canon(x[0] + x[1]);
    cf[1] = canon(mulw(x[1] - x[0] + 3 * Q, w1));
  } else {
    u64 a0 = x[0], a1 = x[1], a2 = x[2], a3 = x[3];
    bf_inv<3>(a0, a1, w3);
    bf_inv<3>(a2, a3, w2);
    cf[0] = canon(a0 + a2);
    cf[1] = canon(a1 + a3);
    cf[2] = canon(mulw(a2 - a0 + 5 * Q, w1));
    cf[3] = canon(mulw(a3 - a1 + 3 * Q, w1));
  }
}

// The forward's first log R stages on one digit of the R coefficients: at most 3 log R.
template <int R>
__device__ __forceinline__ void cross_forward(const u32 (&g)[R], u64 (&y)[R], const Tw& w1, const Tw& w2, const Tw& w3) {
#pragma unroll
  for (int k = 0; k < R / 2; k++) {
    const u64 t = mulw_digit(g[k + R / 2], w1);
    y[k] = g[k] + t;
    y[k + R / 2] = g[k] + 3 * Q - t;
  }
  if constexpr (R == 4) {
    bf_fwd(y[0], y[1], w2);
    bf_fwd(y[2], y[3], w3);
  }
}

// Position of slot t's gathered operands: a warp's lanes (slots 2 l + k) gather from distinct banks, as slot8
// arranges for units of eight.
template <int LOGN>
__device__ __forceinline__ int slot2(int t) {
  return ((t & 1) << (LOGN - 1)) | (t >> 1);
}

// Words between the CTAs of a cluster: st.async stores a word in a CTA's shared memory and counts its bytes
// on an mbarrier there, so a receiver waits for its data alone. A cluster barrier's release made every
// thread wait until its remote stores had landed and its loads were back (1,400 cycles of a 6,480-cycle
// link, twice).
__device__ __forceinline__ u32 cluster_addr(u32 addr, int rank) {
  u32 a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void send_word(u32 to, u64 v, u32 bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to), "l"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void store_remote(u32 to, u64 v) {
  asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(to), "l"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int LOGN, int R>
__global__ void __launch_bounds__((1 << LOGN) / R / 2, 1)
    k_respond_cluster(CrsDev c, const QueryDev* queries, const ShardDev* shards, const u64* b_fold, u64* a_out,
                      u64* b_out, u32* status, int force_serial) {
  namespace cg = cooperative_groups;
  using G = Part<LOGN, R>;
  constexpr int N = G::N, P = G::P, NT = G::NT, LP = G::LP, C = G::C;
  constexpr int TOP = LP & 1 ? LP - 2 : LP - 1;  // bit of the forward's first local pass
  constexpr u32 M2N = 2 * N - 1;
  extern __shared__ __align__(16) u64 sm[];
  u64* XB = sm;           // [R][C] the parts' words that this CTA crosses
  u64* D = XB + P;        // [2][P] this part of digits 0 and 1
  u64* X = D + 2 * P;     // [P] the local inverse
  u64* a_ntt = X + P;
  Tw* fl = reinterpret_cast<Tw*>(a_ntt + N);  // the part's forward ladder
  Tw* il = fl + P;                            // the mirrored part's, for the inverse
  ulonglong2* rows = reinterpret_cast<ulonglong2*>(il + P);  // room for three key rows, as in k_respond
  const KeyRows KR{rows, rows + N, rows + 2 * N};
  uint16_t* s_tab = reinterpret_cast<uint16_t*>(rows + 3 * N);  // position of the slot of exponent 2e + 1

  __shared__ __align__(8) u64 inbox[2];  // arrivals of cross words and of digit words

  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x;
  // Shared memory of the R CTAs (their buffers, then their inboxes).
  const u32 in_words = smem_addr(&inbox[0]), in_digits = smem_addr(&inbox[1]);
  u32 peer[R], peer_words[R], peer_digits[R];
#pragma unroll
  for (int k = 0; k < R; k++) {
    peer[k] = cluster_addr(smem_addr(sm), k);
    peer_words[k] = cluster_addr(in_words, k);
    peer_digits[k] = cluster_addr(in_digits, k);
  }
  if (tid == 0) {
    inbox_init(in_words);
    inbox_init(in_digits);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const QueryDev qd = queries[blockIdx.x / R];
  const u32 qi = qd.row;  // output and status row
  const ShardDev sh = shards[qd.shard];
  const SetView ps = set_view(c, qd.crs);
  const u32 gamma = ps.gamma;

  cluster_arrive();
  if (tid == 0) refuse_stale(sh, status, qi);
  {
#pragma unroll 4
    for (int k = tid; k < N; k += NT) stage_key_rows(ps, qd.seat, KR, N, k, slot2<LOGN>(k));
#pragma unroll 8
    for (int k = tid; k < N; k += NT) s_tab[k] = (uint16_t)slot2<LOGN>(c.exp_slot[k]);
    Tw f[2], i[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int k = max(tid + j * NT, 1);
      f[j] = c.tw[part_ladder<R>(k, rank)];
      i[j] = c.tw[part_ladder<R>(k, R - 1 - rank)];
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      fl[tid + j * NT] = f[j];
      il[tid + j * NT] = i[j];
    }
  }
  const Tw w1 = c.tw[1], w2 = R == 4 ? c.tw[2] : w1, w3 = R == 4 ? c.tw[3] : w1;
  const int base = rank * P, l0 = base + 2 * tid;  // this thread's slots: l0, l0 + 1
  const u32 et[2] = {c.slot_exp[l0], c.slot_exp[l0 + 1]};
  // The query's a, expanded in the exchange buffers' place by every CTA, each transforming its part: the first log R
  // stages of the part's words, its local stages as one digit's. The slots go to every CTA's a_ntt.
  static_assert(4 * P >= N, "a fits the buffers");
  expand_a<N, NT>(qd, sm, status, qi, force_serial);  // ends with a barrier
  {
    u64 y[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const u64* x = sm + tid + j * NT;
      u64 u = x[0], v;
      if constexpr (R == 2) {
        v = mulw(x[P], w1);
      } else {
        const u64 t0 = mulw(x[2 * P], w1), t1 = mulw(x[3 * P], w1);
        u += rank < 2 ? t0 : 3 * Q - t0;
        v = mulw(rank < 2 ? x[P] + t1 : x[P] + 3 * Q - t1, rank < 2 ? w2 : w3);
      }
      y[j] = u + (rank & 1 ? 3 * Q - v : v);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; j++) D[G::sw(tid + j * NT)] = y[j];
    __syncthreads();
    part_forward<LOGN, R, TOP, 7>(D, fl);  // the second buffer's words go along unused
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(D + G::sw(2 * tid));
    u64 a0 = part_bound(LP, TOP, 7) > 12 ? red60(v.x) : v.x, a1 = v.y;
    bf_fwd(a0, a1, fl[P / 2 + tid]);
    a0 = canon(mulw(a0, c.s_ninv_rinv));
    a1 = canon(mulw(a1, c.s_ninv_rinv));
    cluster_wait();  // every CTA runs
#pragma unroll
    for (int k = 0; k < R; k++) {
      const u32 to = peer[k] + (u32)((uint8_t*)a_ntt - (uint8_t*)sm);
      store_remote(to + 8 * slot2<LOGN>(l0), a0);
      store_remote(to + 8 * slot2<LOGN>(l0 + 1), a1);
    }
  }
  cluster.sync();  // every CTA has its a, and is past its use of the exchange buffers
  u64 cur[2];
  Acc sb[2];
  {
    const u32 gp = ps.gpow[gamma - 1];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      cur[k] = mulq(a_ntt[s_tab[((gp * et[k]) & M2N) >> 1]], sh.sums_R[(size_t)(gamma - 1) * N + l0 + k]);
      sb[k] = Acc{0, 0, 0, 0};
    }
  }
  // This thread's cross word and, with four CTAs, its digit.
  const int q = tid & (C - 1), dg = tid / C;
  // Twiddles of the thread's own pair: stage 0 of the inverse, the last of the forward.
  const Tw wi0 = il[P - 1 - tid], wf0 = fl[P / 2 + tid];
  // The thread's pair through the local inverse, its words to the CTAs that cross them (their words buffer, or with
  // `second` their digits').
  auto inverse_to_cross = [&](u64 x0, u64 x1, u32 second) {
    const u32 off = second * 8 * P, box = second * 8;
    bf_inv<2>(x0, x1, wi0);
    *reinterpret_cast<ulonglong2*>(X + G::sw(2 * tid)) = make_ulonglong2(x0, x1);
    __syncthreads();
    part_inverse<LOGN, R, 1>(X, il, [&](int e, int k, u64 x) {
      const u32 at = off + 8 * (rank * C + (e & (C - 1)));
      if constexpr (G::bits(LP & 1 ? LP - 2 : LP - 1) == G::LR) {  // the pass holds the bits of the crossing CTA
        send_word(peer[k] + at, x, peer_words[k] + box);
      } else {
        send_word(cluster_addr(smem_addr(sm) + at, e / C), x, cluster_addr(in_words + box, e / C));
      }
    });
  };
  // A wait that runs out marks the query failed; the links then run on without waiting, to their end.
  bool alive = true;
  u32 parity = 0;  // of the next phase of either inbox
  auto await = [&](u32 bar) {
    if (alive && !inbox_wait(bar, parity)) {
      alive = false;
      atomicOr(status + qi, (u32)DEV_PEER_TIMEOUT);
    }
  };
  auto links = [&](auto gadget) {
    constexpr bool EXACT = decltype(gadget)::value;
    // The online sum's operands of the link before.
    u64 pd0[2] = {0, 0}, pd1[2] = {0, 0}, pc[2] = {0, 0};
    u32 pt[2] = {0, 0};
    auto online = [&](int i) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const ulonglong2 y = KR.Y01[pt[k]];
        mac(sb[k], pd0[k], y.x);
        mac(sb[k], pd1[k], y.y);
        if constexpr (EXACT) mac(sb[k], pc[k], KR.WY2[pt[k]].y);
        if (i % SB_FOLD_LINKS == 0) sb[k] = acc_from(acc_fold(sb[k]));
      }
    };
#pragma unroll 1
    for (int i = (int)gamma - 2; i >= 0; i--) {
      const ulonglong2 sv = *reinterpret_cast<const ulonglong2*>(sh.sums_R + (size_t)i * N + l0);
      const u32 gp = ps.gpow[i];
      if (tid == 0 && alive) {
        inbox_expect(in_words, P * 8);
        inbox_expect(in_digits, 2 * P * 8);
      }
      inverse_to_cross(cur[0], cur[1], 0);
      online(i);
      await(in_words);
      {
        u64 x[R], cf[R], y[R];
#pragma unroll
        for (int k = 0; k < R; k++) x[k] = XB[k * C + q];
        cross_inverse<R>(x, cf, w1, w2, w3);
        u32 g[2][R];
#pragma unroll
        for (int k = 0; k < R; k++) split_digits<EXACT>(cf[k], g[0][k], g[1][k]);
        const int at = G::sw(rank * C + q);
#pragma unroll
        for (int n = 0; n < 2; n++) {
          u32 h[R];
          if constexpr (R == 4) {
            if (n) break;  // one digit a thread
#pragma unroll
            for (int k = 0; k < R; k++) h[k] = dg ? g[1][k] : g[0][k];
          } else {
#pragma unroll
            for (int k = 0; k < R; k++) h[k] = g[n][k];
          }
          cross_forward<R>(h, y, w1, w2, w3);
          const u32 to = 8 * (P + (R == 4 ? dg : n) * P + at);
#pragma unroll
          for (int k = 0; k < R; k++) send_word(peer[k] + to, y[k], peer_digits[k]);
        }
      }
      // What the pointwise step has without the digits, while they travel.
      Acc r[2];
      ulonglong2 w[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const u32 tb = s_tab[((gp * et[k]) & M2N) >> 1];
        w[k] = KR.W01[tb];
        r[k] = Acc{0, 0, 0, 0};
        mac(r[k], a_ntt[tb], k ? sv.y : sv.x);
        if constexpr (EXACT) mac(r[k], cur[k], KR.WY2[tb].x);
        pc[k] = cur[k];
        pt[k] = tb;
      }
      await(in_digits);
      parity ^= 1;
      part_forward<LOGN, R, TOP, 3 * G::LR>(D, fl);
      u64 d[2][2];
#pragma unroll
      for (int n = 0; n < 2; n++) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(D + n * P + G::sw(2 * tid));
        d[n][0] = part_bound(LP, TOP, 3 * G::LR) > 12 ? red60(v.x) : v.x;
        d[n][1] = v.y;
        bf_fwd(d[n][0], d[n][1], wf0);
      }
#pragma unroll
      for (int k = 0; k < 2; k++) {
        mac(r[k], d[0][k], w[k].x);
        mac(r[k], d[1][k], w[k].y);
        pd0[k] = d[0][k];
        pd1[k] = d[1][k];
        cur[k] = acc_fold(r[k]);
      }
    }
    online(0);
  };
  if (ps.approx == 0)
    links(std::true_type{});
  else
    links(std::false_type{});
  // Final inverse transforms of c_0 (to a) and of the online sum (to b): local stages, then the cross. With four CTAs
  // the sum's words go to the digits' buffer (a peer that sent its first words has read its last digits) and the two
  // crosses run side by side, on half the threads each (12,200 -> 8,800 cycles after the links); with two every
  // thread crosses, one transform after the other.
  scan_done();
  constexpr bool SIDE = R == 4;
  auto cross = [&](int n, auto read) {
    u64 x[R], cf[R];
#pragma unroll
    for (int k = 0; k < R; k++) x[k] = XB[(SIDE ? n * P : 0) + k * C + q];
    read();
    // Unscaled residues: finish_a takes the coefficient as it is, finish_b times n^-1.
    cross_inverse<R>(x, cf, w1, w2, w3);
#pragma unroll
    for (int k = 0; k < R; k++) {
      const int t = k * P + rank * C + q;
      if (n == 0)
        a_out[(size_t)qi * N + t] = finish_a(cf[k], qd.ms);
      else
        b_out[(size_t)qi * N + t] = finish_b(c, cf[k], t, gamma, b_fold + qd.fold_off, qd.ms);
    }
  };
#pragma unroll 1
  for (int n = 0; n < 2; n++) {
    const u32 second = SIDE ? n : 0, box = in_words + 8 * second;
    if (tid == 0 && alive) inbox_expect(box, P * 8);
    inverse_to_cross(n ? acc_fold(sb[0]) : cur[0], n ? acc_fold(sb[1]) : cur[1], second);
    await(box);
    if constexpr (!SIDE) {
      parity ^= 1;
      cross(n, [&] { cluster.sync(); });  // the words are read before the next are sent, and before a CTA ends
    } else if (n == 0) {
      // Every thread has read X before the next transform rewrites it. The arrivals alone say so only where each thread of
      // the last local pass sends a word to its own CTA; a pass of one bit (rings 256 and 1024) sends to two CTAs of the four.
      __syncthreads();
    }
  }
  if constexpr (SIDE) {
    cross(dg, [] {});
    cluster.sync();  // no CTA ends with words on their way to a peer
  }
}

// ------------------------------------------------------------------------------------
// NoPacking respond (respond.rs:614-643): one RLWE ciphertext (a h_j, b h_j) per column j
// (plaintext_multiply_columns, respond.rs:585-599) and their sum.
//   nopack_prep: per query, NTT(a) and NTT(b) in R-form (a expanded from the seed);
//   nopack_cols: per (query, column), NTT(h_j), the two products (one Montgomery product
//                each against the R-form operands) and their inverse transforms, written
//                as ciphertext 1 + j of the query;
//   nopack_sum:  ciphertext 0 = the sum of the column ciphertexts mod q.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_nopack_prep(CrsDev c, const QueryDev* queries, Tw r_mod_q,
                                                                 u64* AB_R, u32* status) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  u64* xa = sm;
  u64* xb = sm + N;
  Tw* tw = reinterpret_cast<Tw*>(sm + 2 * N);
  const u32 qi = blockIdx.x;
  const QueryDev qd = queries[qi];
  for (int k = threadIdx.x; k < N; k += NT) {
    tw[k] = c.tw[k];
    xb[k] = reduce128(qd.b[k]);
  }
  expand_a<N, NT>(qd, xa, status, qi, 0);  // ends with a barrier
  {
    u64* const bufs[2] = {xa, xb};
    ntt_fwd_r4<LOGN, NT, 2>(bufs, tw);
  }
  u64* o = AB_R + (size_t)qi * 2 * N;
  for (int k = threadIdx.x; k < N; k += NT) {
    o[k] = canon(mulw(xa[k], r_mod_q));
    o[N + k] = canon(mulw(xb[k], r_mod_q));
  }
}

template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_nopack_cols(CrsDev c, const QueryDev* queries,
                                                                 const ShardDev* shards, const u64* AB_R, u64* out) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  u64* x = sm;
  u64* ya = sm + N;
  u64* yb = sm + 2 * N;
  Tw* tw = reinterpret_cast<Tw*>(sm + 3 * N);
  const u32 j = blockIdx.x, qi = blockIdx.y;
  const QueryDev qd = queries[qi];
  const u64* col = shards[qd.shard].columns + (size_t)j * N;
  for (int k = threadIdx.x; k < N; k += NT) {
    tw[k] = c.tw[k];
    x[k] = reduce128(col[k]);
  }
  __syncthreads();
  {
    u64* const bufs[1] = {x};
    ntt_fwd_r4<LOGN, NT, 1>(bufs, tw);
  }
  const u64* A = AB_R + (size_t)qi * 2 * N;
  for (int k = threadIdx.x; k < N; k += NT) {
    const u64 h = canon(x[k]);
    ya[k] = mont(A[k], h);
    yb[k] = mont(A[N + k], h);
  }
  __syncthreads();
  {
    u64* const bufs[2] = {ya, yb};
    ntt_inv_r4<LOGN, NT, 2>(bufs, tw);
  }
  u64* o = out + ((size_t)qi * (c.gamma + 1) + 1 + j) * 2 * N;
  for (int k = threadIdx.x; k < N; k += NT) {
    o[k] = canon(mulw(ya[k], c.ninv));
    o[N + k] = canon(mulw(yb[k], c.ninv));
  }
}

// A CTA sums 32 words of a query's ciphertexts, a warp every eighth column, eight loads in flight: one thread a word over
// all the columns waited for 256 loads in turn on 16 CTAs a query (39 us for one query of gamma 256).
constexpr int SUM_WARPS = 8;
__global__ void __launch_bounds__(32 * SUM_WARPS) k_nopack_sum(u32 n, u32 gamma, u64* out) {
  __shared__ u64 part[SUM_WARPS][32];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;  // over 2n words
  u64* base = out + (size_t)blockIdx.y * (gamma + 1) * 2 * n + k;
  u64 acc = 0;
#pragma unroll 8
  for (u32 j = 1 + w; j <= gamma; j += SUM_WARPS) acc = addq(acc, base[(size_t)j * 2 * n]);
  part[w][lane] = acc;
  __syncthreads();
  if (w) return;
#pragma unroll
  for (int r = 1; r < SUM_WARPS; r++) acc = addq(acc, part[r][lane]);
  base[0] = acc;
}

// ------------------------------------------------------------------------------------
// OnePacking: respond_one_packing (pir/respond.rs:696-729), the Galois-automorphism tree of
// inspiring/automorph_pack.rs. Leaf j (j < gamma) is the column product's
// a part a h_j (b part zero) and b-value_j = coeff0(b h_j), which the shard scan gives; leaves past gamma are
// the padding's zero ciphertexts. Node (ell, start) = (E + y O) + keyswitch(tau_t(E - y O)) with
// E, O its children (start, start + n/2^ell), y = X^(n >> ell), t = 2^ell + 1 and Galois key
// log n - ell (pack_lwes_inner, automorph_pack.rs:96-163). Every node whose start is at or
// past gamma is exactly zero, so only those below gamma are computed.
//
// Nodes live in the NTT domain, scaled by n^-1 as k_respond's links hold R: y O is a product by NTT(X^s),
// tau_t a slot permutation, and only the key switch's digit split needs coefficients: a = INTT(tau_t(...).a),
// digits 0 and 1 (base 2^20) transformed, digit 2's transform base^-2 (a - D0 - base D1) (the
// unsigned split of rgsw/external_product.rs:58-99 leaves a = D0 + base D1 + base^2 D2
// exactly), which the keys' folded rows (fold_gadget_keys) take from a itself.
//
// The walk is the recursion's depth-first order: leaf k of the walk is start = bitrev(k),
// and a binary-counter carry combines each finished node with its waiting sibling; the
// waiting nodes sit in a stack of node slots in global memory. At gamma < n the odd children of the lowest
// log(n / gamma) levels are all zero: a leaf walks those levels alone, from its registers (three of four nodes at
// gamma 256; with the keys laid out for their loads 64 queries 4.80 -> 3.63 ms). The leaves [j n/S, (j+1) n/S) of
// the walk make up the subtree of start bitrev(j) at level log n - log S, so S CTAs walk a query's subtrees, and of two
// CTAs whose subtrees are siblings the one that ends last goes on with the node above: log S nodes after the last
// subtree (one CTA walking all S - 1 of them took 0.2 ms after a batch's subtrees: 64 queries 3.64 -> 3.51 ms, one
// 0.91 -> 0.37). A query on one CTA took 11 ms whatever the batch, and 64 left most SMs idle. 103 KB of shared memory a CTA: two on an SM.
struct TreeSmem {
  Tw* tw;
  u64 *S1a, *S1b, *D;  // E - y O of a node, by gather position; the transforms' buffers (2N)
  uint16_t* s_tab;     // gather position of the slot of exponent 2e + 1
};
template <int LOGN>
__device__ __forceinline__ TreeSmem tree_stage(const CrsDev& c, u64* sm) {
  constexpr int N = 1 << LOGN, NT = N / 8;
  TreeSmem S{reinterpret_cast<Tw*>(sm), sm + 2 * N, sm + 3 * N, sm + 4 * N, reinterpret_cast<uint16_t*>(sm + 6 * N)};
  for (int k = threadIdx.x; k < N; k += NT) {
    S.tw[tw8<LOGN>(k)] = c.tw[k];
    S.s_tab[k] = (uint16_t)slot8<LOGN>(c.exp_slot[k]);
  }
  return S;
}
// A node in global memory: (a, b) of 2N words, each thread's pairs of slots apart by the thread count.
template <int LOGN>
__device__ __forceinline__ void node_load(const u64* node, u64 (&a)[8], u64 (&b)[8]) {
  constexpr int NT = (1 << LOGN) / 8;
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(node) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const ulonglong2 x = __ldcg(p + k * NT), y = __ldcg(p + (k + 4) * NT);  // another CTA may have written it
    a[2 * k] = x.x, a[2 * k + 1] = x.y, b[2 * k] = y.x, b[2 * k + 1] = y.y;
  }
}
template <int LOGN>
__device__ __forceinline__ void node_store(u64* node, const u64 (&a)[8], const u64 (&b)[8]) {
  constexpr int NT = (1 << LOGN) / 8;
  ulonglong2* p = reinterpret_cast<ulonglong2*>(node) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    p[k * NT] = make_ulonglong2(a[2 * k], a[2 * k + 1]);
    p[(k + 4) * NT] = make_ulonglong2(b[2 * k], b[2 * k + 1]);
  }
}
// The current node (a, b at the thread's slots) becomes (E + y O) + keyswitch(tau_t(E - y O)) at level ell: it is
// O and E waits in memory, or it is E itself, its odd sibling zero (E null). Ends with a barrier.
template <int LOGN>
__device__ __forceinline__ void tree_combine(const CrsDev& c, const TreeSmem& S, const u64* E, int ell,
                                             const u32 (&et)[8], u64 (&ca)[8], u64 (&cb)[8]) {
  constexpr int N = 1 << LOGN, NT = N / 8;
  constexpr u32 M2N = 2 * N - 1;
  const u32 sy = (u32)(N >> ell), t = (1u << ell) + 1;
  if (!E) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      S.S1a[k * NT + threadIdx.x] = ca[k];
      S.S1b[k * NT + threadIdx.x] = cb[k];
    }
  } else {
    u64 ea[8], eb[8];
    node_load<LOGN>(E, ea, eb);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const Tw y = c.pow_root[(et[k] * sy) & M2N];
      const u64 ya = canon(mulw(ca[k], y)), yb = canon(mulw(cb[k], y));
      ca[k] = addq(ea[k], ya);
      cb[k] = addq(eb[k], yb);
      S.S1a[k * NT + threadIdx.x] = subq(ea[k], ya);
      S.S1b[k * NT + threadIdx.x] = subq(eb[k], yb);
    }
  }
  __syncthreads();
  u64 d[2][8];
  {
    u64 aa[8];
#pragma unroll
    for (int k = 0; k < 8; k++) aa[k] = S.S1a[S.s_tab[((t * et[k]) & M2N) >> 1]];
    link_transforms8<LOGN, true>(aa, d, S.D, S.tw);
  }
  const ulonglong2* key = reinterpret_cast<const ulonglong2*>(c.galois + (size_t)(LOGN - ell) * 6 * N) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    ulonglong2 w[6];
#pragma unroll
    for (int r = 0; r < 6; r++) w[r] = key[(r * 4 + k / 2) * NT];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const u32 at = S.s_tab[((t * et[k + j]) & M2N) >> 1];
      const u64 aa = S.S1a[at];
      Acc na{0, 0, 0, 0}, nb{0, 0, 0, 0};
      mac(na, d[0][k + j], j ? w[0].y : w[0].x);
      mac(nb, d[0][k + j], j ? w[1].y : w[1].x);
      mac(na, d[1][k + j], j ? w[2].y : w[2].x);
      mac(nb, d[1][k + j], j ? w[3].y : w[3].x);
      mac(na, aa, j ? w[4].y : w[4].x);
      mac(nb, aa, j ? w[5].y : w[5].x);
      ca[k + j] = addq(ca[k + j], csub(acc_fold(na)));
      cb[k + j] = addq(cb[k + j], addq(S.S1b[at], csub(acc_fold(nb))));
    }
  }
  __syncthreads();  // S1 and D are rewritten next
}

template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8, 2)
    k_tree(CrsDev c, const QueryDev* queries, const ShardDev* shards, u32 log_parts, u64 ms_target, u64* stack, u64* roots,
           u32* arrived, const u64* b_fold, u64* a_out, u64* b_out, u32* status) {
  constexpr int N = 1 << LOGN, NT = N / 8, P = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  const TreeSmem S = tree_stage<LOGN>(c, sm);
  const int tid = threadIdx.x;
  const u32 qi = blockIdx.x >> log_parts, part = blockIdx.x & ((1u << log_parts) - 1);
  const QueryDev qd = queries[qi];
  const ShardDev sh = shards[qd.shard];
  const u32 gamma = c.gamma;
  const int levels = LOGN - (int)log_parts;
  const int zeros = LOGN - (31 - __clz(gamma));  // levels whose odd children are all zero
  u64* stk = stack + (size_t)blockIdx.x * (levels - zeros) * 2 * N;
  u64* slots = roots + ((size_t)qi << log_parts) * 2 * N;
  __shared__ u32 first;
  u32 et[8];
  u64 aR[8];  // n^-1 NTT(a) at the thread's slots
#pragma unroll
  for (int k = 0; k < 8; k++) et[k] = c.slot_exp[8 * tid + k];
  expand_a<N, NT>(qd, S.D + N, status, qi, 0);  // ends with a barrier
  transform_slots8<LOGN>(S.D + N, S.D, S.tw, c.ninv, aR);
  u64 ca[8], cb[8];
#pragma unroll 1
  for (u32 m = 0;; m++) {
    const u32 start = __brev((part << levels) | (m << zeros)) >> (32 - LOGN);
    {
      // Leaf `start`: the column through the transform times NTT(a).
      __syncthreads();  // every thread is past its last read of D
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int b = tid + r * NT;
        u64 x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const size_t at = (size_t)start * N + b + j * P;
          x[j] = sh.cols16 ? (u64)sh.cols16[at] : red60(sh.columns[at]);
        }
        fwd_unit<false>(x[0], x[1], x[2], x[3], S.tw[1], S.tw[2], S.tw[3]);
#pragma unroll
        for (int j = 0; j < 4; j++) S.D[sw8(b + j * P)] = x[j];
      }
      __syncthreads();
      fwd_middle8<LOGN, 1, 7>(S.D, S.tw);
      u64 x[1][8];
      fwd_last8<LOGN, 1, fwd_bound8(LOGN, 2, 7)>(x, S.D, S.tw);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        ca[j] = csub(mulq(x[0][j], aR[j]));
        cb[j] = 0;
      }
    }
    if (gamma == 1) break;  // a single leaf is the root
    bool root = false;
#pragma unroll 1
    for (int L = 0;; L++) {
      const u64* E = nullptr;
      if (L >= levels) {
        // Above the subtrees a node waits in the slot of its first subtree; the first of two siblings to arrive leaves,
        // the other goes on. The even one is E whichever comes last.
        const u32 up = L - levels, at = part >> up;
        if (up == log_parts) {
          root = true;
          break;
        }
        u64 *mine = slots + ((size_t)at << up) * 2 * N, *other = slots + ((size_t)(at ^ 1) << up) * 2 * N;
        node_store<LOGN>(mine, ca, cb);
        __threadfence();
        __syncthreads();
        if (tid == 0) first = atomicAdd(arrived + (qi << log_parts) + (1u << (log_parts - 1 - up)) + (at >> 1), 1u) == 0;
        __syncthreads();
        if (first) return;
        __threadfence();
        if (!(at & 1)) node_load<LOGN>(other, ca, cb);
        E = at & 1 ? other : mine;
      } else if (L >= zeros) {
        u64* wait = stk + (size_t)(L - zeros) * 2 * N;
        if (!((m >> (L - zeros)) & 1)) {
          node_store<LOGN>(wait, ca, cb);
          break;
        }
        E = wait;
      }
      tree_combine<LOGN>(c, S, E, L + 1, et, ca, cb);
    }
    if (root) break;
  }
  // The root to coefficients; b_z += n b-value_z for z < gamma (pack_lwes, automorph_pack.rs 327-338), except for a
  // single input, which pack_lwes returns untouched: no tree and no d scaling.
  scan_done();
  inv_first8<LOGN>(ca, S.D, S.tw);
  inv_first8<LOGN>(cb, S.D + N, S.tw);
  __syncthreads();
  inv_middle8<LOGN, 2>(S.D, S.tw);
  const u64* bval = b_fold + queries[qi].fold_off;
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int b = tid + r * NT;
#pragma unroll
    for (int n = 0; n < 2; n++) {
      u64 x[4];
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = S.D[n * N + sw8(b + k * P)];
      inv_unit(x[0], x[1], x[2], x[3], S.tw[3], S.tw[2], S.tw[1]);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const u32 z = b + k * P;
        u64 v = canon(x[k]);
        if (n == 1) {
          if (gamma == 1)
            v = z == 0 ? bval[0] : 0;
          else if (z < gamma)
            v = addq(v, reduce128(wide(bval[z], (u64)N)));
        }
        if (ms_target) v = mod_switch_word(v, ms_target);
        (n ? b_out : a_out)[(size_t)qi * N + z] = v;
      }
    }
  }
}

// ------------------------------------------------------------------------------------
// Client side (ClientSession::query_batch, session.rs:377-434; extract_inspiring and
// extract_packed, extract.rs:184-263): queries and record decoding for many queries at once.
//
// The query error comes from the session's Gaussian sampler (math/gaussian.rs:210-224),
// one stream shared by the whole batch in order: each sample draws x uniform in
// [-tailcut, tailcut] (rand's widening-multiply rejection: a 64-bit word whose low product
// half exceeds the zone is skipped) and then u uniform in [0, 1) from one 64-bit word, and
// keeps x when threshold(x) > bits(u). Read as a machine over the stream's 64-bit words it
// has two states, A (next word is an x candidate) and B (next word is the u of an accepted
// x), so the stream is parsed in parallel: each thread composes the state maps of a segment
// of words, a scan gives every segment its start state, and a second walk counts and places
// the samples.

// Word i of the stream: u32 words base + 2i, base + 2i + 1 of the keystream buffer.
__device__ __forceinline__ u64 ks_word(const u32* ks, u64 base, u64 i) {
  return (u64)ks[base + 2 * i] | ((u64)ks[base + 2 * i + 1] << 32);
}
// x of candidate word w, or false when rand rejects it.
__device__ __forceinline__ bool gauss_x(const GaussDev& g, u64 w, i64& x) {
  const u128 m = (u128)w * g.range;
  if ((u64)m > g.zone) return false;
  x = -g.tailcut + (i64)(u64)(m >> 64);
  return true;
}
// rand's f64 in [0, 1) from w (52 high bits as the mantissa of [1, 2), minus 1, exact), and
// the acceptance of x: threshold bits above the bits of u.
__device__ __forceinline__ bool gauss_keep(const GaussDev& g, i64 x, u64 w) {
  const double v = __longlong_as_double((long long)((w >> 12) | 0x3FF0000000000000ULL)) - 1.0;
  return g.accept[x + g.tailcut] > (u64)__double_as_longlong(v);
}

// The sampler's keystream: ChaCha20 blocks block0 .. block0 + nblocks - 1 of stream 0.
__global__ void k_keystream(const u32* key, u64 block0, u64 nblocks, u32* ks) {
  const u64 b = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nblocks) return;
  u32 k[8], out[16];
#pragma unroll
  for (int i = 0; i < 8; i++) k[i] = key[i];
  chacha20_block(k, block0 + b, 0, out);
#pragma unroll
  for (int i = 0; i < 16; i++) ks[b * 16 + i] = out[i];
}

// Segment t (words [t seg, t seg + seg) of W): bit 0 = end state from A, bit 1 = from B.
__global__ void k_gauss_maps(GaussDev g, const u32* ks, u64 base, u64 W, u32 seg, uint8_t* maps, u64 T) {
  const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  u32 sa = 0, sb = 1;
  const u64 e = min(W, (t + 1) * seg);
  for (u64 i = t * seg; i < e; i++) {
    i64 x;
    const u32 next_a = gauss_x(g, ks_word(ks, base, i), x) ? 1u : 0u;
    sa = sa ? 0u : next_a;
    sb = sb ? 0u : next_a;
  }
  maps[t] = (uint8_t)(sa | (sb << 1));
}

// One block: exclusive scan of T segment maps from state A (start states), or, with
// counts, exclusive prefix sums of T counts (offsets) and their total.
__global__ void __launch_bounds__(1024) k_gauss_scan(const uint8_t* maps, uint8_t* starts, const u32* counts,
                                                     u64* offsets, u64* total, u64 T) {
  __shared__ u64 part[1024];
  const u64 per = (T + 1023) / 1024;
  const u64 b = threadIdx.x * per, e = min(T, b + per);
  if (maps) {
    // Composite map of this thread's range, as the pair (image of A, image of B).
    u32 fa = 0, fb = 1;
    for (u64 i = b; i < e; i++) {
      const u32 m = maps[i];
      fa = (m >> fa) & 1;
      fb = (m >> fb) & 1;
    }
    part[threadIdx.x] = fa | (fb << 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      u32 st = 0;
      for (int c = 0; c < 1024; c++) {
        const u32 m = (u32)part[c];
        part[c] = st;
        st = (m >> st) & 1;
      }
    }
    __syncthreads();
    u32 st = (u32)part[threadIdx.x];
    for (u64 i = b; i < e; i++) {
      starts[i] = (uint8_t)st;
      st = (maps[i] >> st) & 1;
    }
  } else {
    u64 sum = 0;
    for (u64 i = b; i < e; i++) sum += counts[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      u64 acc = 0;
      for (int c = 0; c < 1024; c++) {
        const u64 v = part[c];
        part[c] = acc;
        acc += v;
      }
      *total = acc;
    }
    __syncthreads();
    u64 acc = part[threadIdx.x];
    for (u64 i = b; i < e; i++) {
      offsets[i] = acc;
      acc += counts[i];
    }
  }
}

// Walk of segment t from its start state: counts its samples (offsets null), or writes
// sample k to out[k] for k < S and, at the S-th, the word index after it to *end.
__global__ void k_gauss_walk(GaussDev g, const u32* ks, u64 base, u64 W, u32 seg, const uint8_t* starts, u64 T,
                             u32* counts, const u64* offsets, u64 S, i64* out, u64* end) {
  const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  u64 i = t * seg;
  const u64 e = min(W, i + seg);
  u32 st = starts[t];
  i64 x = 0;
  if (st == 1) gauss_x(g, ks_word(ks, base, i - 1), x);  // the pending x is the previous word's
  u64 k = offsets ? offsets[t] : 0;
  u32 n = 0;
  for (; i < e; i++) {
    const u64 w = ks_word(ks, base, i);
    if (st == 0) {
      st = gauss_x(g, w, x) ? 1u : 0u;
    } else {
      st = 0;
      if (gauss_keep(g, x, w)) {
        if (offsets) {
          if (k < S) out[k] = x;
          if (k == S - 1) *end = i + 1;
          k++;
        } else {
          n++;
        }
      }
    }
  }
  if (!offsets) counts[t] = n;
}

// One CTA per query: b = Delta X^-local - a s + e (SeededRgswCiphertext::encrypt_with_rng,
// rgsw/types.rs:345-388, one gadget row of power 1), a from the query's seed.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_client_query(CrsDev c, const QueryDev* queries,
                                                                  const u64* s_R, const u32* locals,
                                                                  const i64* samples, u64 delta, u64* b_out,
                                                                  u32* status) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  Tw* tw = reinterpret_cast<Tw*>(sm);
  u64* x = sm + 2 * N;
  const u32 qi = blockIdx.x;
  const QueryDev qd = queries[qi];
  for (int k = threadIdx.x; k < N; k += NT) {
    tw[k] = c.tw[k];
  }
  expand_a<N, NT>(qd, x, status, qi, 0);  // ends with a barrier
  {
    u64* const bufs[1] = {x};
    ntt_fwd_r4<LOGN, NT, 1>(bufs, tw);
  }
  for (int k = threadIdx.x; k < N; k += NT) x[k] = mont(canon(x[k]), s_R[k]);
  __syncthreads();
  {
    u64* const bufs[1] = {x};
    ntt_inv_r4<LOGN, NT, 1>(bufs, tw);
  }
  const u32 local = locals[qi];
  const int pos = local == 0 ? 0 : N - (int)local;
  const u64 mono = local == 0 ? delta : Q - delta;  // Delta X^-local (encode_db.rs:43-70)
  for (int k = threadIdx.x; k < N; k += NT) {
    const u64 as = canon(mulw(x[k], c.ninv));
    const i64 ev = samples[(size_t)qi * N + k];
    u64 b = addq(negq(as), ev < 0 ? Q - (u64)(-ev) : (u64)ev);
    if (k == pos) b = addq(b, mono);
    b_out[(size_t)qi * N + k] = b;
  }
}

// One CTA per response: (a s + b) mod the response modulus, rounded by delta and taken mod p
// (PlaintextRounding, rlwe/enc.rs:14-44); times d^-1 mod p for a tree response; the first
// ceil(entry/2) values are the record's 16-bit columns (encode_db.rs:152-168). The product
// is taken mod q: a switched modulus m keeps |a s| below n m max|s| < q/2, so the centred
// residue is the integer product (the host checks the bound).
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_client_extract(CrsDev c, const u64* s_R, const u64* a,
                                                                    const u64* b, u64 modulus, u64 delta, u64 p,
                                                                    u64 dinv, u32 entry_size, uint8_t* out) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  extern __shared__ __align__(16) u64 sm[];
  Tw* tw = reinterpret_cast<Tw*>(sm);
  u64* x = sm + 2 * N;
  const u32 qi = blockIdx.x;
  for (int k = threadIdx.x; k < N; k += NT) {
    tw[k] = c.tw[k];
    x[k] = a[(size_t)qi * N + k];
  }
  __syncthreads();
  {
    u64* const bufs[1] = {x};
    ntt_fwd_r4<LOGN, NT, 1>(bufs, tw);
  }
  for (int k = threadIdx.x; k < N; k += NT) x[k] = mont(canon(x[k]), s_R[k]);
  __syncthreads();
  {
    u64* const bufs[1] = {x};
    ntt_inv_r4<LOGN, NT, 1>(bufs, tw);
  }
  const u32 cols = (entry_size + 1) / 2;
  for (u32 k = threadIdx.x; k < cols && k < (u32)N; k += NT) {
    u64 as = canon(mulw(x[k], c.ninv));
    if (modulus != Q) {
      const bool neg = as > (Q >> 1);
      const u64 mag = (neg ? Q - as : as) % modulus;
      as = neg && mag ? modulus - mag : mag;
    }
    const u64 bv = b[(size_t)qi * N + k];
    u64 noisy = as + bv;
    if (noisy >= modulus) noisy -= modulus;
    u64 m = ((noisy + delta / 2) / delta) % p;
    if (dinv) m = (u64)((u128)m * dinv % p);
    uint8_t* rec = out + (size_t)qi * entry_size;
    rec[2 * k] = (uint8_t)(m & 0xff);
    if (2 * k + 1 < entry_size) rec[2 * k + 1] = (uint8_t)((m >> 8) & 0xff);
  }
}

// ------------------------------------------------------------------------------------
// Integer roofline probe: the recursion kernels' lazy forward butterflies (bf_fwd: one product by
// a twiddle and two 64-bit sums, the transforms' unit of work) on values held in registers, eight
// per thread, no memory traffic. Its rate is the ceiling the respond kernels' butterflies are
// measured against.
__global__ void __launch_bounds__(256) k_butterfly_peak(u64* out, int iters, Tw w) {
  u64 x[8];
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = (u64)(blockIdx.x * 8191u + threadIdx.x * 131u + k) * 0x9E3779B97F4A7C15ULL % Q;
#pragma unroll 1
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) bf_fwd(x[k], x[k + 1], w);
#pragma unroll
    for (int k = 0; k < 4; k++) bf_fwd(x[k], x[k + 4], w);
  }
  u64 acc = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) acc ^= x[k];
  if (acc == 0x123456789ULL) out[0] = acc;  // keeps the chains live; practically never taken
}

// ------------------------------------------------------------------------------------
// Launchers.

#define IG_DISPATCH_LOGN(logn, ...)                   \
  switch (logn) {                                     \
    case 8: { constexpr int L = 8; __VA_ARGS__; } break;   \
    case 9: { constexpr int L = 9; __VA_ARGS__; } break;   \
    case 10: { constexpr int L = 10; __VA_ARGS__; } break; \
    case 11: { constexpr int L = 11; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;                 \
  }

cudaError_t fold_gadget_keys(const CrsDev& c, const u64* keys, u64* out, u32 count, cudaStream_t s) {
  const u32 total = count * 2 * c.n;
  if (total == 0) return cudaSuccess;
  k_fold_gadget_keys<<<(total + 255) / 256, 256, 0, s>>>(c, keys, out, count);
  return cudaGetLastError();
}

cudaError_t key_rows(const CrsDev& c, const u64* in, u64* out, u32 rows, const KeyScale& f, cudaStream_t s) {
  if (rows != 2 && rows != 3) return cudaErrorInvalidValue;
  const size_t smem = 3 * (size_t)c.n * 8;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = rows;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(rows);
  cfg.blockDim = dim3(c.n / 4);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = rows == 3 ? k_key_rows<L, 3> : k_key_rows<L, 2>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k, c, in, out, f);
    if (e != cudaSuccess) return e;
  });
  return cudaGetLastError();
}

cudaError_t ntt_rows(const CrsDev& c, const u64* in, u64* out, u32 rows, u64 scale, cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  const size_t smem = 3 * (size_t)c.n * 8;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_ntt_rows<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<rows, (1 << L) / 4, smem, s>>>(c, in, out, make_tw(scale));
  });
  return cudaGetLastError();
}

static cudaError_t store_sums(const CrsDev& c, const ShardArg& shards, u32 count, u64* H, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  if (c.gamma > (u32)FOLD_TILE || c.gamma == 0 || c.gamma > c.n) return cudaErrorInvalidValue;
  u32 SL = FOLD_TILE / c.gamma;
  if (SL > c.n) SL = c.n;
  if (c.n % SL) return cudaErrorInvalidValue;
  const size_t smem_ntt = 3 * (size_t)c.n * 8;
  const u32 lgs = 31 - __builtin_clz(SL);
  const size_t smem_fold = (fold_twiddles(c.gamma) + 8) * sizeof(Tw) + c.n * 2 + (size_t)SL * (c.gamma + 1) * 8;
  IG_DISPATCH_LOGN(c.logn, {
    auto kn = k_store_ntt<L>;
    cudaError_t e = cudaFuncSetAttribute(kn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_ntt);
    if (e != cudaSuccess) return e;
    kn<<<dim3((c.gamma + STORE_ROWS - 1) / STORE_ROWS, count), (1 << L) / 8, smem_ntt, s>>>(c, shards, H);
  });
  using Fold = void (*)(CrsDev, const u64*, ShardArg, u32);
  static constexpr Fold folds[] = {k_store_fold<0>, k_store_fold<1>, k_store_fold<2>, k_store_fold<3>,
                                   k_store_fold<4>, k_store_fold<5>, k_store_fold<6>, k_store_fold<7>,
                                   k_store_fold<8>, k_store_fold<9>, k_store_fold<10>};
  const u32 lg = 31 - __builtin_clz(c.gamma);
  if (lg >= sizeof folds / sizeof folds[0]) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(folds[lg], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_fold);
  if (e != cudaSuccess) return e;
  folds[lg]<<<dim3(c.n / SL, count), FOLD_THREADS, smem_fold, s>>>(c, H, shards, lgs);
  return cudaGetLastError();
}
cudaError_t store_sums(const CrsDev& c, const ShardDev* table, u32 count, u64* H, cudaStream_t s) {
  return store_sums(c, ShardArg{table, {}}, count, H, s);
}
cudaError_t store_sums_one(const CrsDev& c, const ShardDev& shard, u64* H, cudaStream_t s) {
  return store_sums(c, ShardArg{nullptr, shard}, 1, H, s);
}

u32 scan_chunks(u32 gamma) { return (gamma + SCAN_COLS - 1) / SCAN_COLS; }

cudaError_t shard_scan(const CrsDev& c, const QueryDev* queries, const ShardDev* shards, u32 nq, const u32* work,
                       u32 nwork, u64* b_fold, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  const u32 chunks = scan_chunks(c.gamma);
  const u32 blocks = work ? nwork : nq * chunks;
  if (blocks == 0) return cudaSuccess;
  const size_t smem = scan_smem_bytes((int)c.n);
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_scan<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<blocks, SCAN_WARPS * 32, smem, s>>>(c, queries, shards, work, chunks, b_fold);
  });
  return cudaGetLastError();
}

cudaError_t tag_keys(const CrsDev& c, const ShardDev* table, u32 count, const u32 (&seed)[8], u64 stream, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  TagSeed t;
  for (int k = 0; k < 8; k++) t.w[k] = seed[k];
  k_tag_keys<<<dim3((c.n / 4 + 127) / 128, count), 128, 0, s>>>(c.n, table, t, stream);
  return cudaGetLastError();
}

cudaError_t column_tags(const CrsDev& c, const ShardDev* table, u32 count, bool any_wide, u32* mismatch, cudaStream_t s) {
  if (c.gamma == 0 || count == 0) return cudaSuccess;
  constexpr u32 per_cta = 8;  // warps of 256 threads, one column each
  const size_t smem = scan_smem_bytes((int)c.n);
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_column_tags16<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<dim3(scan_chunks(c.gamma), count), SCAN_WARPS * 32, smem, s>>>(c.gamma, table, mismatch);
    if (any_wide)
      k_column_tags<L><<<dim3((c.gamma + per_cta - 1) / per_cta, count), per_cta * 32, 0, s>>>(c.gamma, table, mismatch);
  });
  return cudaGetLastError();
}

cudaError_t encode_records(const uint8_t* rec, u64 entries, u32 entry_size, u32 n, u32 gamma, const ShardDev* table,
                           u32 count, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  k_encode_records<<<dim3((gamma + ENC_COLS - 1) / ENC_COLS, n / ENC_ROWS, count), 256, 0, s>>>(rec, entries, entry_size, n,
                                                                                            gamma, table);
  return cudaGetLastError();
}

cudaError_t wire(const u64* a, const u64* b, u32 count, u32 n, u32 retained, u32 bits, u64 modulus,
                 const uint8_t* tmpl, u32 len, u32 a_off, u32 a_bytes, u32 b_off, u32 b_bytes, uint8_t* out,
                 u32* status, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  dim3 grid((len + 255) / 256, count);
  k_wire<<<grid, 256, 0, s>>>(a, b, n, retained, bits, modulus, tmpl, len, a_off, a_bytes, b_off, b_bytes, out,
                              status);
  return cudaGetLastError();
}

cudaError_t compact16(const u64* cols, size_t words, uint16_t* out, u32* wide, cudaStream_t s) {
  if (words == 0 || words % 8) return cudaErrorInvalidValue;
  const size_t groups = words / 8;
  const unsigned threads = 256;
  k_compact16<<<(unsigned)((groups + threads - 1) / threads), threads, 0, s>>>(cols, groups, out, wide);
  return cudaGetLastError();
}

cudaError_t nopack_prep(const CrsDev& c, const QueryDev* queries, u32 nq, u64 r_mod_q, u64* AB_R, u32* status,
                        cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  const size_t smem = 4 * (size_t)c.n * 8;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_nopack_prep<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<nq, (1 << L) / 4, smem, s>>>(c, queries, make_tw(r_mod_q), AB_R, status);
  });
  return cudaGetLastError();
}

cudaError_t nopack_cols(const CrsDev& c, const QueryDev* queries, const ShardDev* shards, u32 nq, const u64* AB_R,
                        u64* out, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  const size_t smem = 5 * (size_t)c.n * 8;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_nopack_cols<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<dim3(c.gamma, nq), (1 << L) / 4, smem, s>>>(c, queries, shards, AB_R, out);
  });
  k_nopack_sum<<<dim3(2 * c.n / 32, nq), 32 * SUM_WARPS, 0, s>>>(c.n, c.gamma, out);
  return cudaGetLastError();
}

cudaError_t keystream(const u32* key, u64 block0, u64 nblocks, u32* ks, cudaStream_t s) {
  if (nblocks == 0) return cudaSuccess;
  k_keystream<<<(unsigned)((nblocks + 255) / 256), 256, 0, s>>>(key, block0, nblocks, ks);
  return cudaGetLastError();
}

cudaError_t gauss_parse(const GaussDev& g, const u32* ks, u64 base, u64 W, u32 seg, uint8_t* maps, uint8_t* starts,
                        u32* counts, u64* offsets, u64* total, u64 S, i64* out, u64* end, cudaStream_t s) {
  const u64 T = (W + seg - 1) / seg;
  const unsigned blocks = (unsigned)((T + 255) / 256);
  k_gauss_maps<<<blocks, 256, 0, s>>>(g, ks, base, W, seg, maps, T);
  k_gauss_scan<<<1, 1024, 0, s>>>(maps, starts, nullptr, nullptr, nullptr, T);
  k_gauss_walk<<<blocks, 256, 0, s>>>(g, ks, base, W, seg, starts, T, counts, nullptr, S, out, end);
  k_gauss_scan<<<1, 1024, 0, s>>>(nullptr, nullptr, counts, offsets, total, T);
  k_gauss_walk<<<blocks, 256, 0, s>>>(g, ks, base, W, seg, starts, T, nullptr, offsets, S, out, end);
  return cudaGetLastError();
}

cudaError_t client_query(const CrsDev& c, const QueryDev* queries, u32 nq, const u64* s_R, const u32* locals,
                         const i64* samples, u64 delta, u64* b_out, u32* status, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  const size_t smem = 3 * (size_t)c.n * 8;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_client_query<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<nq, (1 << L) / 4, smem, s>>>(c, queries, s_R, locals, samples, delta, b_out, status);
  });
  return cudaGetLastError();
}

cudaError_t client_extract(const CrsDev& c, u32 count, const u64* s_R, const u64* a, const u64* b, u64 modulus,
                           u64 delta, u64 p, u64 dinv, u32 entry_size, uint8_t* out, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  const size_t smem = 3 * (size_t)c.n * 8;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_client_extract<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<count, (1 << L) / 4, smem, s>>>(c, s_R, a, b, modulus, delta, p, dinv, entry_size, out);
  });
  return cudaGetLastError();
}

// Subtrees of a query (a power of two): the split that takes least by a model in key switches (a leaf counts as
// one; 10.2 us on an SM alone), with the stacks and roots within 256 MB. A subtree takes its own length on an idle
// GPU; a full one gets through the batch's work at 1.2 subtrees an SM (two CTAs share it), with half a
// subtree of idle tail; log S nodes above follow. Measured at gamma 256 (ms, 4 / 8 / 32 subtrees): a query alone
// 2.24 / 1.17 / 0.37, 64 queries 3.97 / 3.93 / 3.49 (16 subtrees 3.48), 152 7.76 / 7.82 / 7.87.
u32 tree_log_parts(const CrsDev& c, u32 nq, u32 sms) {
  u64 work = c.gamma, best = ~0ULL;  // leaves and nodes of a whole tree
  for (u32 k = 1; k <= c.logn; k++) work += c.gamma < (c.n >> k) ? c.gamma : c.n >> k;
  u32 log_best = 0;
  for (u32 lp = 0; lp <= 5 && (2u << lp) <= c.gamma; lp++) {
    if (lp && tree_scratch_words(c, nq, lp) * 8 > (256ULL << 20)) break;
    const u64 part = work >> lp, full = nq * work * 10 / (12 * (u64)sms) + part / 2;
    const u64 cost = (part > full ? part : full) + lp;
    if (cost < best) best = cost, log_best = lp;
  }
  return log_best;
}
// Node stacks of the subtrees, then their roots' slots.
static u64 tree_stack_words(const CrsDev& c, u32 nq, u32 log_parts) {
  return ((u64)nq << log_parts) * (31 - __builtin_clz(c.gamma) - log_parts) * 2 * c.n;
}
u64 tree_scratch_words(const CrsDev& c, u32 nq, u32 log_parts) {
  return tree_stack_words(c, nq, log_parts) + ((u64)nq << log_parts) * 2 * c.n;
}

cudaError_t tree(const CrsDev& c, const QueryDev* queries, const ShardDev* shards, u32 nq, u32 log_parts, u64 ms_target,
                 u64* nodes, u32* arrived, const u64* b_fold, u64* a_out, u64* b_out, u32* status, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  if (!c.galois || c.gamma > c.n / 2) return cudaErrorInvalidValue;
  const size_t smem = (size_t)6 * c.n * 8 + 2 * (size_t)c.n;
  u64* roots = nodes + tree_stack_words(c, nq, log_parts);
  // Beside the scan before it: only a query's last CTA takes its folds (scan_done).
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nq << log_parts);
  cfg.blockDim = dim3(c.n / 8);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = k_tree<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaLaunchKernelEx(&cfg, k, c, queries, shards, log_parts, ms_target, nodes, roots, arrived, b_fold, a_out, b_out,
                             status);
    if (e != cudaSuccess) return e;
  });
  return cudaGetLastError();
}

cudaError_t butterfly_peak(u64* out, int blocks, int iters, cudaStream_t s) {
  const u64 w = 0x0123456789ABCDEULL % Q;
  k_butterfly_peak<<<blocks, 256, 0, s>>>(out, iters, make_tw(w));
  return cudaGetLastError();
}

size_t respond_smem_bytes(const CrsDev& c, int ctas) {
  // Transform buffers (2n words, or four parts of n / ctas), a_ntt and the ladder, three key rows of W and Y, the
  // u16 slot table.
  const size_t n = c.n;
  const size_t words = ctas == 1 ? 2 * n + 3 * n + 6 * n : 4 * n / ctas + n + 4 * n / ctas + 6 * n;
  return words * 8 + n * 2;
}

u32 max_quads() {
  CrsDev c{};
  c.n = 2048;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 4;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(4);
  cfg.blockDim = dim3(c.n / 8);
  cfg.dynamicSmemBytes = respond_smem_bytes(c, 4);
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  auto k = k_respond_cluster<11, 4>;
  int n = 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return (u32)n;
}

cudaError_t respond(const CrsDev& c, const QueryDev* queries, const ShardDev* shards, u32 nq,
                    const u64* b_fold, u64* a_out, u64* b_out, u32* status,
                    int force_serial_expand, int ctas, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  if (ctas != 1 && ctas != 2 && ctas != 4) return cudaErrorInvalidValue;
  const size_t smem = respond_smem_bytes(c, ctas);
  // A cluster a query, and a start beside the scan before it on the stream (the scan lets its successor launch at once,
  // the recursion reads the folds only at its end: scan_done). The recursion's CTAs fill the SMs that the scan's last
  // wave leaves: a lone query of gamma 16 142 -> 131 us, 128 mixed queries 5.20 -> 5.00 ms, 64 of one shard
  // 1.47 -> 1.46 ms.
  cudaLaunchAttribute attrs[2]{};
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = (unsigned)ctas;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas * nq);
  cfg.blockDim = dim3(ctas == 1 ? c.n / 8 : c.n / ctas / 2);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attrs;
  cfg.numAttrs = ctas == 1 ? 1 : 2;
  IG_DISPATCH_LOGN(c.logn, {
    auto k = ctas == 4 ? k_respond_cluster<L, 4> : ctas == 2 ? k_respond_cluster<L, 2> : k_respond<L>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k, c, queries, shards, b_fold, a_out, b_out, status, force_serial_expand);
    if (e != cudaSuccess) return e;
  });
  return cudaGetLastError();
}


}  // namespace igk
