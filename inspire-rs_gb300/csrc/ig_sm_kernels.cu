// Kernels of the special_modulus respond path (reference src/special_modulus/server.rs).
//
//   ntt_rows      forward Ntt32 of many rows (seat limbs, key mask, table columns)
//   table_columns nibble decode of a shard's cells (mod.rs:366-371, server.rs:211-249)
//   table_fold    step 1 folded over the columns (server.rs:331-383) as a per-slot DFT
//   body_fold     the response body's column fold over the shard's nibbles (server.rs:401-411)
//   respond       the 2n-link two-prime recursion and final transforms (server.rs:386-498)
//
// Every word is a canonical residue; products are Montgomery with R = 2^32 as in Prime32.
#include <cuda_runtime.h>

#include <type_traits>

#include "ig_arith.cuh"
#include "ig_sm.cuh"

namespace igsmk {
using namespace igsm;

// ------------------------------------------------------------------------------------
// Forward Ntt32 in shared memory, radix-4 (one 4-word unit per thread, N/4 threads). The stage
// schedule and twiddle indices are those of arith.rs:169-251: Cooley-Tukey over fwd[m + i].
template <int LOGN>
__device__ __forceinline__ void fwd32(u32* x, const Ntt32Dev& T, const u32* tw) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  static_assert(LOGN & 1, "odd log n: one radix-2 stage then radix-4 pairs");
  const Prime32 P = T.p;
  const int tid = threadIdx.x;
  {
    constexpr int t = N / 2;
    const u32 w = tw[1];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int b = tid + r * NT;
      const u32 u = x[b], v = P.mont(x[b + t], w);
      x[b] = P.add(u, v);
      x[b + t] = P.sub(u, v);
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int s = 1; s < LOGN; s += 2) {
    const int t = N >> (s + 1), m = 1 << s, h = t >> 1;
    const int i = tid / h, o = tid - i * h;
    const int e0 = i * 2 * t + o;
    const u32 wa = tw[m + i], wb = tw[2 * m + 2 * i], wc = tw[2 * m + 2 * i + 1];
    u32 a0 = x[e0], a1 = x[e0 + h], a2 = x[e0 + t], a3 = x[e0 + t + h];
    u32 v = P.mont(a2, wa);
    a2 = P.sub(a0, v);
    a0 = P.add(a0, v);
    v = P.mont(a3, wa);
    a3 = P.sub(a1, v);
    a1 = P.add(a1, v);
    v = P.mont(a1, wb);
    x[e0] = P.add(a0, v);
    x[e0 + h] = P.sub(a0, v);
    v = P.mont(a3, wc);
    x[e0 + t] = P.add(a2, v);
    x[e0 + t + h] = P.sub(a2, v);
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4) k_sm_ntt_rows(SmDev c, int which, const u32* in, u32* out,
                                                                 int to_mont) {
  constexpr int N = 1 << LOGN, NT = N / 4;
  __shared__ u32 x[N];
  __shared__ u32 tw[N];
  const Ntt32Dev& T = which ? c.lp : c.lq;
  const u32* row = in + (size_t)blockIdx.x * N;
  for (int k = threadIdx.x; k < N; k += NT) {
    x[k] = row[k] % T.p.m;
    tw[k] = T.fwd[k];
  }
  __syncthreads();
  fwd32<LOGN>(x, T, tw);
  // to_mont: mont(x, 2^64 mod m) = x 2^32 mod m.
  const u32 r2 = (u32)((((unsigned __int128)1) << 64) % T.p.m);
  u32* o = out + (size_t)blockIdx.x * N;
  for (int k = threadIdx.x; k < N; k += NT) o[k] = to_mont ? T.p.mont(x[k], r2) : x[k];
}

// values[m][j] for m < n (zero past `rows`), colq[j][m] = the nibble as a residue mod q.
__global__ void k_sm_columns(SmDev c, const uint8_t* cells, u32 rows, u32 cell_bytes, int8_t* values, u32* colq) {
  const u32 idx = blockIdx.x * blockDim.x + threadIdx.x;  // over n rows x gamma/2 bytes
  const u32 half = c.gamma / 2;
  if (idx >= c.n * half) return;
  const u32 m = idx / half, byte = idx % half;
  const uint8_t b = m < rows && byte < cell_bytes ? cells[(size_t)m * cell_bytes + byte] : 0;
  const int8_t lo = (int8_t)((int8_t)(uint8_t)(b << 4) >> 4);
  const int8_t hi = (int8_t)((int8_t)b >> 4);
  values[(size_t)m * c.gamma + 2 * byte] = lo;
  values[(size_t)m * c.gamma + 2 * byte + 1] = hi;
  colq[(size_t)(2 * byte) * c.n + m] = c.lq.p.small(lo);
  colq[(size_t)(2 * byte + 1) * c.n + m] = c.lq.p.small(hi);
}

// Step 1 per slot t (root w_t = w0^e_t): acc_i[t] = sum_j w_t^(j c_i) H_j[t] with
// c_i = g^-i = 1 + m_i (2n/gamma), i.e. a length-gamma DFT of u_j = w0^(e_t j) H_j[t] read
// at (e_t m_i) mod gamma; then S_i[t'] = gamma^-1 acc_i[t] at the slot t' whose image under
// tau_{g^i} is t, in R-form.
constexpr int SM_FOLD_TILE = 2048;
constexpr int SM_FOLD_THREADS = 256;

template <int LOGN>
__global__ void __launch_bounds__(SM_FOLD_THREADS) k_sm_fold(SmDev c, const u32* H, u32* step1_R, u32 SL) {
  constexpr int N = 1 << LOGN;
  constexpr u32 M2N = 2 * N - 1;
  __shared__ u32 x[SM_FOLD_TILE];
  __shared__ u32 pw[2 * N];
  const u32 gamma = c.gamma, tile = SL * gamma, t0 = blockIdx.x * SL;
  const Prime32 P = c.lq.p;
  u32 lg = 0;
  while ((1u << lg) < gamma) lg++;
  for (int k = threadIdx.x; k < 2 * N; k += SM_FOLD_THREADS) pw[k] = c.pow_root_R[k];
  __syncthreads();
  for (u32 idx = threadIdx.x; idx < tile; idx += SM_FOLD_THREADS) {
    const u32 j = idx / SL, s = idx % SL;
    const u32 e = c.slot_exp[t0 + s];
    x[s * gamma + j] = P.mont(H[(size_t)j * N + t0 + s], pw[(e * j) & M2N]);
  }
  __syncthreads();
  for (u32 len = gamma >> 1; len >= 1; len >>= 1) {
    for (u32 b = threadIdx.x; b < SL * (gamma >> 1); b += SM_FOLD_THREADS) {
      const u32 s = b / (gamma >> 1), bb = b % (gamma >> 1);
      const u32 blk = bb / len, j = bb % len;
      const u32 i0 = s * gamma + blk * 2 * len + j;
      const u32 u = x[i0], v = x[i0 + len];
      x[i0] = P.add(u, v);
      x[i0 + len] = P.mont(P.sub(u, v), pw[(j * (N / len)) & M2N]);
    }
    __syncthreads();
  }
  for (u32 idx = threadIdx.x; idx < tile; idx += SM_FOLD_THREADS) {
    const u32 i = idx / SL, s = idx % SL;
    const u32 e = c.slot_exp[t0 + s];
    const u32 k = (e * c.m_of_i[i]) & (gamma - 1);
    const u32 kr = lg ? (__brev(k) >> (32 - lg)) : 0;
    const u32 tp = c.exp_slot[((c.cpow[i] * e) & M2N) >> 1];
    step1_R[(size_t)i * N + tp] = P.mont(x[s * gamma + kr], c.inv_gamma_RR);
  }
}

// ------------------------------------------------------------------------------------
// Body fold: fold[chunk][k] = sum c_m values[m][k] over the rows of one of SM_FOLD_CHUNKS chunks of the shard (exact
// in i64; the respond kernel adds the chunks). A thread takes eight columns (all of them below gamma 8) of every eighth
// row, one 64-bit load a row. The chunk's c_m are staged as their low 16 bits and the rest, so a product is two
// 32-bit multiply-adds, which sum exactly over a thread's rows (at most 64: 2^16 2^7 2^6 < 2^31), where a 64-bit sum
// took a wide multiply and a 64-bit add. A CTA a query walking all rows byte by byte took 377 us for 256 queries of
// 1 MB of nibbles each, four columns a thread on 64-bit sums 150 us
// (the call 4.02 -> 3.96 ms).
constexpr int SM_FOLD_ROWS = 8, SM_FOLD_COLS = 8, SM_FOLD_SPAN = 512;  // rows side by side, columns a thread, rows a chunk
__global__ void __launch_bounds__(512) k_sm_body_fold(SmDev c, const SmQueryDev* queries, i64* fold) {
  __shared__ i64 part[SM_FOLD_ROWS - 1][512];
  __shared__ int2 cm[SM_FOLD_SPAN];
  // The respond launch that follows may start now: it takes the folds only at its end.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const SmQueryDev qd = queries[blockIdx.x];
  const u32 cols = min(c.gamma, (u32)SM_FOLD_COLS);
  const u32 lanes = blockDim.x / SM_FOLD_ROWS, k0 = threadIdx.x % lanes * cols, r0 = threadIdx.x / lanes;
  const u32 span = (qd.rows + SM_FOLD_CHUNKS - 1) / SM_FOLD_CHUNKS;
  const u32 from = min(qd.rows, blockIdx.y * span), rows = min(qd.rows, from + span) - from;
  const Prime32 P = c.lq.p;
  for (u32 r = threadIdx.x; r < rows; r += blockDim.x) {
    const u32 m = from + r, bw = qd.body[m == 0 ? 0 : c.n - m];
    const int x = (int)(m == 0 ? P.centred(bw) : -P.centred(bw));
    cm[r] = make_int2(x & 0xffff, x >> 16);
  }
  __syncthreads();
  int lo[SM_FOLD_COLS] = {}, hi[SM_FOLD_COLS] = {};
  const int8_t* base = qd.values + (size_t)from * c.gamma + k0;
#pragma unroll 8
  for (u32 r = r0; r < rows; r += SM_FOLD_ROWS) {
    const int2 x = cm[r];
    const int8_t* row = base + (size_t)r * c.gamma;
    uint2 v = make_uint2(0, 0);
    if (cols == 8)
      v = *reinterpret_cast<const uint2*>(row);
    else if (cols == 4)
      v.x = *reinterpret_cast<const u32*>(row);
    else  // two columns
      v.x = *reinterpret_cast<const uint16_t*>(row);
#pragma unroll
    for (int j = 0; j < SM_FOLD_COLS; j++) {
      const int n = (int)(int8_t)((j < 4 ? v.x : v.y) >> (8 * (j & 3)));
      lo[j] += x.x * n;
      hi[j] += x.y * n;
    }
  }
  i64 acc[SM_FOLD_COLS];
#pragma unroll
  for (int j = 0; j < SM_FOLD_COLS; j++) {
    acc[j] = (i64)hi[j] * 65536 + lo[j];
    if (r0 && j < (int)cols) part[r0 - 1][k0 + j] = acc[j];
  }
  __syncthreads();
  if (r0) return;
  i64* out = fold + ((size_t)blockIdx.x * SM_FOLD_CHUNKS + blockIdx.y) * c.gamma + k0;
#pragma unroll
  for (int j = 0; j < SM_FOLD_COLS; j++) {
    if (j >= (int)cols) break;
    for (int r = 0; r < SM_FOLD_ROWS - 1; r++) acc[j] += part[r][k0 + j];
    out[j] = acc[j];
  }
}

// ------------------------------------------------------------------------------------
// expand_uniform (mod.rs:225-237) on the query seed's stream 0: accept u < floor(2^64/q) q,
// take u mod q. Word w of the stream is keystream words 2w, 2w+1. A rejection (probability
// below 2^-35 per word) shifts the rest, and the walk is redone word by word.
template <int N, int NT>
__device__ __forceinline__ void sm_expand(const SmQueryDev& qd, u32 q, u32* a, u32* status, u32 qi) {
  const int tid = threadIdx.x;
  const u64 zone = (~0ULL / q) * q;
  bool rejected = false;
  u32 key[8];
#pragma unroll
  for (int k = 0; k < 8; k++) key[k] = qd.seed[k];
  if (tid < N / 8) {
    u32 blk[16];
    ig::chacha20_block(key, (u64)tid, 0, blk);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const u64 v = (u64)blk[2 * k] | ((u64)blk[2 * k + 1] << 32);
      if (v >= zone) rejected = true;
      a[tid * 8 + k] = (u32)(v % q);
    }
  }
  if (__syncthreads_or(rejected)) {
    if (tid == 0) {
      u32 blk[16];
      u64 have = ~0ULL, cand = 0;
      int filled = 0;
      const u64 limit = (u64)N + 65536;
      while (filled < N && cand < limit) {
        const u64 bi = cand >> 3;
        if (bi != have) {
          ig::chacha20_block(key, bi, 0, blk);
          have = bi;
        }
        const int k = (int)(cand & 7);
        const u64 v = (u64)blk[2 * k] | ((u64)blk[2 * k + 1] << 32);
        if (v < zone) a[filled++] = (u32)(v % q);
        cand++;
      }
      if (filled < N) {
        atomicOr(status + qi, 2u);
        for (; filled < N; filled++) a[filled] = 0;
      }
    }
    __syncthreads();
  }
}

// p_to_q_centred / q_to_p_centred (mod.rs:334-355).
__device__ __forceinline__ u32 p_to_q(const SmDev& c, u32 r) {
  const Prime32 Q = c.lq.p;
  u32 base = r;
  for (u32 k = 0; k < c.p_over_q; k++) base = Q.csub(base);
  return r > (c.lp.p.m >> 1) ? Q.add(base, c.neg_off) : base;
}
// The same lift left in [0, 3q) for the lazy q passes: one Barrett step (the quotient
// estimate from floor(2^32 / q) is the true quotient or one less, r being below 2^32)
// leaves r mod q plus at most q, and the centred offset adds less than q.
__device__ __forceinline__ u32 p_to_q_lazy(const SmDev& c, u32 r) {
  const u32 base = r - __umulhi(r, c.q_mu) * c.lq.p.m;
  return r > (c.lp.p.m >> 1) ? base + c.neg_off : base;
}
__device__ __forceinline__ u32 q_to_p(const SmDev& c, u32 x) {
  return x > (c.lq.p.m >> 1) ? x + (c.lp.p.m - c.lq.p.m) : x;
}

// ------------------------------------------------------------------------------------
// Radix-8 transforms of the recursion: N/8 threads, three stages a shared-memory round trip, layouts free of bank
// conflicts (32-bit words, 32 to a bank row): sw spreads the 16-byte accesses of contiguous units (bit 5 into
// bit 2) and the stride-8 passes (bits 6-7 into 3-4); the ladders' top two levels hold the entries that a unit
// takes N/8 apart; gathered operands sit at (t & 7) N/8 + (t >> 3).
//
// Twiddle products are Shoup products against the forward ladder's (w, w') pairs. The inverse takes the same
// ladder at the mirrored index: psi^-brv(m) = -psi^brv(3 2^s - 1 - m) for m in [2^s, 2^(s+1)), so
// (X - Y) w^-1 = (Y - X) f.
__device__ __forceinline__ int sw(int e) { return e ^ (((e >> 5) & 1) << 2) ^ (((e >> 6) & 3) << 3); }
template <int LOGN>
__device__ __forceinline__ int ladder_at(int m) {
  constexpr int N = 1 << LOGN, E = N / 8;
  if (m >= N / 2) return N / 2 + (m & 3) * E + ((m - N / 2) >> 2);
  if (m >= N / 4) return N / 4 + (m & 1) * E + ((m - N / 4) >> 1);
  return m;
}
template <int LOGN>
__device__ __forceinline__ int slot_at(int t) {
  return ((t & 7) << (LOGN - 3)) | (t >> 3);
}

// Butterflies of a limb. Full, for a prime below 2^31: the inverse's words are residues, the forward's stay below
// 2m (X is brought below m where it is used). Lazy, for 8m <= 2^32: products stay in [0, 2m), the inverse's words
// below 4m and the forward's below 8m inside a unit and 6m between; RED marks the sums that would pass that.
struct FullLimb {
  Prime32 P;
  template <bool RED>
  __device__ __forceinline__ void fwd(u32& X, u32& Y, uint2 w) const {
    const u32 x = P.csub(X), v = P.shoup(Y, w.x, w.y);
    X = x + v;
    Y = x + P.m - v;
  }
  template <bool RED>
  __device__ __forceinline__ void inv(u32& X, u32& Y, uint2 f) const {
    const u32 d = Y + P.m - X;
    X = P.add(X, Y);
    Y = P.shoup(d, f.x, f.y);
  }
  __device__ __forceinline__ u32 residue_inv(u32 x) const { return x; }
  __device__ __forceinline__ u32 residue_fwd(u32 x) const { return P.csub(x); }
};
struct LazyLimb {
  Prime32 P;
  template <bool RED>
  __device__ __forceinline__ void fwd(u32& X, u32& Y, uint2 w) const {
    const u32 x = RED ? csub_by(X, 4 * P.m) : X, v = P.shoupl(Y, w.x, w.y);
    X = x + v;
    Y = x + 2 * P.m - v;
  }
  template <bool RED>
  __device__ __forceinline__ void inv(u32& X, u32& Y, uint2 f) const {
    const u32 d = Y + 4 * P.m - X, t = X + Y;
    X = RED ? csub_by(t, 4 * P.m) : t;
    Y = P.shoupl(d, f.x, f.y);
  }
  __device__ __forceinline__ u32 residue_inv(u32 x) const { return P.csub(csub_by(x, 2 * P.m)); }  // below 4m
  __device__ __forceinline__ u32 residue_fwd(u32 x) const { return residue_inv(csub_by(x, 4 * P.m)); }
};

template <class L>
__device__ __forceinline__ void fwd_unit8(const L& l, u32 (&x)[8], uint2 w0, const uint2 (&w1)[2], const uint2 (&w2)[4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) l.template fwd<false>(x[k], x[k + 4], w0);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    l.template fwd<true>(x[k], x[k + 2], w1[0]);
    l.template fwd<true>(x[k + 4], x[k + 6], w1[1]);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) l.template fwd<true>(x[2 * k], x[2 * k + 1], w2[k]);
}
template <class L>
__device__ __forceinline__ void inv_unit8(const L& l, u32 (&x)[8], const uint2 (&f0)[4], const uint2 (&f1)[2], uint2 f2) {
#pragma unroll
  for (int k = 0; k < 4; k++) l.template inv<true>(x[2 * k], x[2 * k + 1], f0[k]);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    l.template inv<true>(x[4 * k], x[4 * k + 2], f1[k]);
    l.template inv<false>(x[4 * k + 1], x[4 * k + 3], f1[k]);  // products below 2m
  }
  l.template inv<true>(x[0], x[4], f2);
  l.template inv<true>(x[1], x[5], f2);
  l.template inv<false>(x[2], x[6], f2);
  l.template inv<false>(x[3], x[7], f2);
}

// Inverse stages 0-2 of thread tid's unit, from registers to buf.
template <int LOGN, class L>
__device__ __forceinline__ void inv_first8(const L& l, u32 (&x)[8], u32* buf, const uint2* tw) {
  constexpr int N = 1 << LOGN, E = N / 8;
  const int tid = threadIdx.x, r = E - 1 - tid;
  uint2 f0[4], f1[2];
#pragma unroll
  for (int j = 0; j < 4; j++) f0[j] = tw[N / 2 + (3 - j) * E + r];
#pragma unroll
  for (int j = 0; j < 2; j++) f1[j] = tw[N / 4 + (1 - j) * E + r];
  inv_unit8(l, x, f0, f1, tw[E + r]);
#pragma unroll
  for (int k = 0; k < 8; k += 4)
    *reinterpret_cast<uint4*>(buf + sw(8 * tid + k)) = make_uint4(x[k], x[k + 1], x[k + 2], x[k + 3]);
}
// Inverse stages S .. logn-3 (a multiple of three), a barrier after each pass.
template <int LOGN, int S, class L>
__device__ __forceinline__ void inv_middle8(const L& l, u32* buf, const uint2* tw) {
  constexpr int N = 1 << LOGN;
  if constexpr (S < LOGN - 2) {
    constexpr int t = 1 << S, M = N >> (S + 1);
    const int B = threadIdx.x >> S, e0 = B * 8 * t + (threadIdx.x & (t - 1));
    uint2 f0[4], f1[2];
#pragma unroll
    for (int j = 0; j < 4; j++) f0[j] = tw[2 * M - 1 - 4 * B - j];
#pragma unroll
    for (int j = 0; j < 2; j++) f1[j] = tw[M - 1 - 2 * B - j];
    u32 x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = buf[sw(e0 + k * t)];
    inv_unit8(l, x, f0, f1, tw[M / 2 - 1 - B]);
#pragma unroll
    for (int k = 0; k < 8; k++) buf[sw(e0 + k * t)] = x[k];
    __syncthreads();
    inv_middle8<LOGN, S + 3>(l, buf, tw);
  }
}
// Forward stages S .. logn-4, a barrier after each pass.
template <int LOGN, int S, class L>
__device__ __forceinline__ void fwd_middle8(const L& l, u32* buf, const uint2* tw) {
  constexpr int N = 1 << LOGN;
  if constexpr (S < LOGN - 3) {
    constexpr int m = 1 << S, h = N >> (S + 3);
    const int i = threadIdx.x / h, e0 = i * 8 * h + threadIdx.x % h;
    uint2 w1[2], w2[4];
#pragma unroll
    for (int j = 0; j < 2; j++) w1[j] = tw[2 * m + 2 * i + j];
#pragma unroll
    for (int j = 0; j < 4; j++) w2[j] = tw[4 * m + 4 * i + j];
    u32 x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = buf[sw(e0 + k * h)];
    fwd_unit8(l, x, tw[m + i], w1, w2);
#pragma unroll
    for (int k = 0; k < 8; k++) buf[sw(e0 + k * h)] = x[k];
    __syncthreads();
    fwd_middle8<LOGN, S + 3>(l, buf, tw);
  }
}
// The last three forward stages of thread tid's unit, to registers.
template <int LOGN, class L>
__device__ __forceinline__ void fwd_last8(const L& l, u32 (&x)[8], const u32* buf, const uint2* tw) {
  constexpr int N = 1 << LOGN, E = N / 8;
  const int tid = threadIdx.x;
  uint2 w1[2], w2[4];
#pragma unroll
  for (int j = 0; j < 2; j++) w1[j] = tw[N / 4 + j * E + tid];
#pragma unroll
  for (int j = 0; j < 4; j++) w2[j] = tw[N / 2 + j * E + tid];
#pragma unroll
  for (int k = 0; k < 8; k += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(buf + sw(8 * tid + k));
    x[k] = v.x, x[k + 1] = v.y, x[k + 2] = v.z, x[k + 3] = v.w;
  }
  fwd_unit8(l, x, tw[E + tid], w1, w2);
}
// The inverse's last two stages on words b + k N/4, the forward's first two.
template <class L>
__device__ __forceinline__ void inv_cross(const L& l, u32 (&x)[4], uint2 w1, uint2 w2, uint2 w3) {
  l.template inv<true>(x[0], x[1], w3);
  l.template inv<true>(x[2], x[3], w2);
  l.template inv<true>(x[0], x[2], w1);
  l.template inv<true>(x[1], x[3], w1);
}
template <class L>
__device__ __forceinline__ void fwd_cross(const L& l, u32 (&x)[4], uint2 w1, uint2 w2, uint2 w3) {
  l.template fwd<false>(x[0], x[2], w1);
  l.template fwd<false>(x[1], x[3], w1);
  l.template fwd<true>(x[0], x[1], w2);
  l.template fwd<true>(x[2], x[3], w3);
}

// One CTA of N/8 threads per query, two on an SM. Each link i = gamma-2 .. 0 (server.rs:434-487):
//   tp = NTT_p(lift(INTT_q(R_{i+1})));  cp = INTT_p(tp . w_p[tau_i]);  rq = NTT_q(lift(cp));
//   R_i = a[tau_i] S_i + (R_{i+1} w_q[tau_i] - rq) / p;
//   acc_q += R_{i+1} key_q[tau_i];  acc_p += tp key_p[tau_i].
// Thread u owns slots 8u..8u+7. Its unit's stages run in registers beside the pointwise steps; each inverse's last
// two stages, the limb lift and the next forward's first two are one pass in place over the words b + k N/4.
// The kernel holds c_i = n^-1 R_i, so the inverses need no 1/n: a and w_q are scaled by n^-1 and 1/p, w_p by n^-1
// and key_q by n when they are staged, rq takes one product by 1/(n p).
//
// Against radix-4 passes on N/4 threads: 12 barriers a link instead of 20, under half the shared-memory
// wavefronts (7,240 a link, a third of them bank conflicts, filled 65% of the time), no product by 1/n.
template <int LOGN, bool LAZY>
__global__ void __launch_bounds__((1 << LOGN) / 8, 2)
    k_sm_respond(SmDev c, const SmQueryDev* queries, const i64* fold, u32* mask_out, u32* body_out, u32* status) {
  constexpr int N = 1 << LOGN, NT = N / 8, P4 = N / 4;
  constexpr u32 M2N = 2 * N - 1;
  using QLimb = std::conditional_t<LAZY, LazyLimb, FullLimb>;
  extern __shared__ __align__(16) u32 smw[];
  u32* buf = smw;
  u32* a = smw + N;                                    // n^-1 a, by gather position
  uint4* keys = reinterpret_cast<uint4*>(smw + 2 * N);  // n key_q, w_q / p, key_p, w_p / n (R-form), by position
  uint2* fq = reinterpret_cast<uint2*>(smw + 6 * N);   // forward ladders with Shoup companions
  uint2* fp = reinterpret_cast<uint2*>(smw + 8 * N);
  uint16_t* s_tab = reinterpret_cast<uint16_t*>(smw + 10 * N);
  const int tid = threadIdx.x;
  const u32 qi = blockIdx.x;
  const SmQueryDev qd = queries[qi];
  const Prime32 PQ = c.lq.p, PP = c.lp.p;
  const QLimb lq{PQ};
  const FullLimb lp{PP};
  for (int k = tid; k < N; k += NT) {
    keys[slot_at<LOGN>(k)] =
        make_uint4(PQ.mont(qd.seat[k], c.n_R), PQ.mont(qd.seat[2 * N + k], c.p_inv_R), qd.seat[N + k],
                   PP.mont(qd.seat[3 * N + k], c.lp.n_inv));
    fq[ladder_at<LOGN>(k)] = c.lq.fwd_sh[k];
    fp[ladder_at<LOGN>(k)] = c.lp.fwd_sh[k];
    s_tab[k] = (uint16_t)slot_at<LOGN>(c.exp_slot[k]);
  }
  sm_expand<N, NT>(qd, PQ.m, buf, status, qi);  // ends with a barrier
  const uint2 wq1 = fq[1], wq2 = fq[2], wq3 = fq[3], wp1 = fp[1], wp2 = fp[2], wp3 = fp[3];
  {
    u32 y[2][4];  // read before any is rewritten at its swizzled place
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int k = 0; k < 4; k++) y[r][k] = buf[tid + r * NT + k * P4];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
      fwd_cross(lq, y[r], wq1, wq2, wq3);
#pragma unroll
      for (int k = 0; k < 4; k++) buf[sw(tid + r * NT + k * P4)] = y[r][k];
    }
    __syncthreads();
    fwd_middle8<LOGN, 2>(lq, buf, fq);
    u32 x[8];
    fwd_last8<LOGN>(lq, x, buf, fq);
#pragma unroll
    for (int k = 0; k < 8; k++) a[k * NT + tid] = PQ.mont(lq.residue_fwd(x[k]), c.lq.n_inv);
    __syncthreads();
  }
  const int l0 = 8 * tid;
  u32 cur[8], accq[8], accp[8], et[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    et[k] = c.slot_exp[l0 + k];
    const u32 tb = s_tab[((c.gpow[c.gamma - 1] * et[k]) & M2N) >> 1];
    cur[k] = PQ.mont(a[tb], qd.step1_R[(size_t)(c.gamma - 1) * N + l0 + k]);
    accq[k] = 0;
    accp[k] = 0;
  }
#pragma unroll 1
  for (int i = (int)c.gamma - 2; i >= 0; i--) {
    const uint4* Srow = reinterpret_cast<const uint4*>(qd.step1_R + (size_t)i * N + l0);
    const uint4 s0 = Srow[0], s1 = Srow[1];
    const u32 gp = c.gpow[i];
    {
      u32 x[8];
#pragma unroll
      for (int k = 0; k < 8; k++) x[k] = cur[k];
      inv_first8<LOGN>(lq, x, buf, fq);
    }
    __syncthreads();
    inv_middle8<LOGN, 3>(lq, buf, fq);
    // INTT_q's end, the lift to p (of residues), NTT_p's start.
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int b = tid + r * NT;
      u32 x[4];
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = buf[sw(b + k * P4)];
      inv_cross(lq, x, wq1, wq2, wq3);
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = q_to_p(c, lq.residue_inv(x[k]));
      fwd_cross(lp, x, wp1, wp2, wp3);
#pragma unroll
      for (int k = 0; k < 4; k++) buf[sw(b + k * P4)] = x[k];
    }
    __syncthreads();
    fwd_middle8<LOGN, 2>(lp, buf, fp);
    {
      u32 tp[8];
      fwd_last8<LOGN>(lp, tp, buf, fp);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint4 key = keys[s_tab[((gp * et[k]) & M2N) >> 1]];
        accp[k] = PP.add(accp[k], PP.mont(tp[k], key.z));
        tp[k] = PP.mont(tp[k], key.w);
      }
      inv_first8<LOGN>(lp, tp, buf, fp);
    }
    __syncthreads();
    inv_middle8<LOGN, 3>(lp, buf, fp);
    // INTT_p's end, the lift to q, NTT_q's start.
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int b = tid + r * NT;
      u32 x[4];
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = buf[sw(b + k * P4)];
      inv_cross(lp, x, wp1, wp2, wp3);
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = LAZY ? p_to_q_lazy(c, x[k]) : p_to_q(c, x[k]);
      fwd_cross(lq, x, wq1, wq2, wq3);
#pragma unroll
      for (int k = 0; k < 4; k++) buf[sw(b + k * P4)] = x[k];
    }
    __syncthreads();
    fwd_middle8<LOGN, 2>(lq, buf, fq);
    u32 rq[8];
    fwd_last8<LOGN>(lq, rq, buf, fq);
    const u32 sv[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const u32 tb = s_tab[((gp * et[k]) & M2N) >> 1];
      const uint2 key = *reinterpret_cast<const uint2*>(keys + tb);
      if constexpr (LAZY) {
        // Products below 2q each: c_i = n^-1 a S + c_{i+1} w_q / p - rq / (n p) below 6q, brought below 4q.
        accq[k] = csub_by(accq[k] + PQ.montl(cur[k], key.x), 2 * PQ.m);
        cur[k] = csub_by(PQ.montl(a[tb], sv[k]) + PQ.montl(cur[k], key.y) + 2 * PQ.m -
                             PQ.shoupl(rq[k], c.np_inv_s, c.np_inv_sp),
                         4 * PQ.m);
      } else {
        accq[k] = PQ.add(accq[k], PQ.mont(cur[k], key.x));
        cur[k] = PQ.add(PQ.mont(a[tb], sv[k]),
                        PQ.sub(PQ.mont(cur[k], key.y), PQ.shoup(rq[k], c.np_inv_s, c.np_inv_sp)));
      }
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the folds of the launch before, which ran beside the links
  // mask = INTT_q(R_0); body = mod_down(INTT_q(acc_q), INTT_p(acc_p)) + fold. No thread touches another's unit
  // of buf before the first barrier of a transform.
  u32 xq[2][4];
#pragma unroll 1
  for (int part = 0; part < 3; part++) {
    u32 x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = part == 0 ? cur[k] : part == 1 ? accq[k] : accp[k];
    if (part < 2) {
      inv_first8<LOGN>(lq, x, buf, fq);
      __syncthreads();
      inv_middle8<LOGN, 3>(lq, buf, fq);
    } else {
      inv_first8<LOGN>(lp, x, buf, fp);
      __syncthreads();
      inv_middle8<LOGN, 3>(lp, buf, fp);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int b = tid + r * NT;
      u32 y[4];
#pragma unroll
      for (int k = 0; k < 4; k++) y[k] = buf[sw(b + k * P4)];
      if (part < 2)
        inv_cross(lq, y, wq1, wq2, wq3);
      else
        inv_cross(lp, y, wp1, wp2, wp3);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int t = b + k * P4;
        if (part == 0) {
          mask_out[(size_t)qi * N + t] = lq.residue_inv(y[k]);
        } else if (part == 1) {
          xq[r][k] = PQ.mont(lq.residue_inv(y[k]), c.lq.n_inv);
        } else if ((u32)t < c.nb) {
          const u32 down = PQ.mont(PQ.sub(xq[r][k], p_to_q(c, PP.mont(y[k], c.lp.n_inv))), c.p_inv_R);
          const i64* chunk = fold + (size_t)qi * SM_FOLD_CHUNKS * c.gamma + t;
          i64 f = 0;
          for (int j = 0; j < SM_FOLD_CHUNKS; j++) f += chunk[j * c.gamma];
          f %= (i64)PQ.m;
          if (f < 0) f += PQ.m;
          body_out[(size_t)qi * c.nb + t] = PQ.add(down, (u32)f);
        }
      }
    }
    __syncthreads();  // buf is rewritten by the next part
  }
}

// ------------------------------------------------------------------------------------
cudaError_t ntt_rows(const SmDev& c, int which, const u32* in, u32* out, u32 rows, int to_mont, cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  if (c.logn != 11) return cudaErrorInvalidValue;
  k_sm_ntt_rows<11><<<rows, 512, 0, s>>>(c, which, in, out, to_mont);
  return cudaGetLastError();
}

cudaError_t table_columns(const SmDev& c, const uint8_t* cells, u32 rows, u32 cell_bytes, int8_t* values, u32* colq,
                          cudaStream_t s) {
  const u32 total = c.n * (c.gamma / 2);
  k_sm_columns<<<(total + 255) / 256, 256, 0, s>>>(c, cells, rows, cell_bytes, values, colq);
  return cudaGetLastError();
}

cudaError_t table_fold(const SmDev& c, const u32* H, u32* step1_R, cudaStream_t s) {
  if (c.logn != 11 || c.gamma == 0 || c.gamma > (u32)SM_FOLD_TILE) return cudaErrorInvalidValue;
  u32 SL = SM_FOLD_TILE / c.gamma;
  if (SL > c.n) SL = c.n;
  k_sm_fold<11><<<c.n / SL, SM_FOLD_THREADS, 0, s>>>(c, H, step1_R, SL);
  return cudaGetLastError();
}

cudaError_t body_fold(const SmDev& c, const SmQueryDev* queries, u32 nq, i64* fold, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  if (c.nb > 512) return cudaErrorInvalidValue;
  // Only the first nb columns reach a response: 512 at most.
  static_assert(SM_FOLD_SPAN * SM_FOLD_CHUNKS >= 2048, "a chunk's rows fit its staging");
  const u32 lanes = c.gamma < SM_FOLD_COLS ? 1 : (c.gamma < 512 ? c.gamma : 512) / SM_FOLD_COLS;
  k_sm_body_fold<<<dim3(nq, SM_FOLD_CHUNKS), SM_FOLD_ROWS * lanes, 0, s>>>(c, queries, fold);
  return cudaGetLastError();
}

cudaError_t respond(const SmDev& c, const SmQueryDev* queries, u32 nq, const i64* fold, u32* mask_out, u32* body_out,
                    u32* status, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  if (c.logn != 11) return cudaErrorInvalidValue;
  const size_t smem = (10 * (size_t)c.n) * 4 + (size_t)c.n * 2;
  // The lazy q-limb passes need every value below 8q to fit 32 bits.
  const bool lazy = (u64)c.lq.p.m * 8 <= (1ULL << 32);
  auto kern = lazy ? k_sm_respond<11, true> : k_sm_respond<11, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // Beside the body fold before it on the stream, whose CTAs leave the SMs one by one (256 queries 4.065 -> 4.033 ms).
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nq);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, c, queries, fold, mask_out, body_out, status);
}

}  // namespace igsmk
