// Poseidon2 over KoalaBear, width 24: initial external layer, 3 full rounds,
// 21 partial rounds (S-box on lane 0), 3 full rounds, S-box x^3
// (recursion/p2_air.go:206-300).  External layer circ(2 M4, M4, ...) with
// gnark-crypto's addition chain for M4 (recursion/p2_air.go:80-104);
// internal layer 1.1^T + diag (recursion/p2_air.go:107-117).
//
// The same code serves the kernels (state in registers, keys in constant
// memory) and the host transcript.
#pragma once
#include "field.cuh"
#include "p2_constants.h"

namespace lg {

static const uint32_t P2_FULL_RK_H[6][24] = LG_P2_FULL_RK_INIT;
static const uint32_t P2_PARTIAL_RK_H[21] = LG_P2_PARTIAL_RK_INIT;
static const uint32_t P2_DIAG_H[24] = LG_P2_DIAG_INIT;
#ifdef __CUDACC__
__constant__ uint32_t P2_FULL_RK_D[6][24] = LG_P2_FULL_RK_INIT;
__constant__ uint32_t P2_PARTIAL_RK_D[21] = LG_P2_PARTIAL_RK_INIT;
#endif

#ifdef __CUDA_ARCH__
#define LG_P2_FULL_RK P2_FULL_RK_D
#define LG_P2_PARTIAL_RK P2_PARTIAL_RK_D
#else
#define LG_P2_FULL_RK P2_FULL_RK_H
#define LG_P2_PARTIAL_RK P2_PARTIAL_RK_H
#endif

LG_HD void p2_m4(uint32_t& x0, uint32_t& x1, uint32_t& x2, uint32_t& x3) {
  uint32_t t01 = add(x0, x1), t23 = add(x2, x3), t0123 = add(t01, t23);
  uint32_t t01123 = add(t0123, x1), t01233 = add(t0123, x3);
  uint32_t y3 = add(dbl(x0), t01233);
  uint32_t y1 = add(dbl(x2), t01123);
  x0 = add(t01, t01123);
  x2 = add(t23, t01233);
  x1 = y1;
  x3 = y3;
}

LG_HD void p2_external(uint32_t s[24]) {
#pragma unroll
  for (int c = 0; c < 6; c++) p2_m4(s[4 * c], s[4 * c + 1], s[4 * c + 2], s[4 * c + 3]);
  uint32_t t0 = s[0], t1 = s[1], t2 = s[2], t3 = s[3];
#pragma unroll
  for (int c = 1; c < 6; c++) {
    t0 = add(t0, s[4 * c]); t1 = add(t1, s[4 * c + 1]);
    t2 = add(t2, s[4 * c + 2]); t3 = add(t3, s[4 * c + 3]);
  }
#pragma unroll
  for (int c = 0; c < 6; c++) {
    s[4 * c] = add(s[4 * c], t0); s[4 * c + 1] = add(s[4 * c + 1], t1);
    s[4 * c + 2] = add(s[4 * c + 2], t2); s[4 * c + 3] = add(s[4 * c + 3], t3);
  }
}

LG_HD uint32_t p2_cube(uint32_t x) { return mul(mul_lazy(x, x), x); }

// The round loops stay rolled: a fully unrolled permutation is more code than
// the SM's instruction caches hold when warps drift apart.
#define LG_PRAGMA(x) _Pragma(#x)
#define LG_UNROLL(n) LG_PRAGMA(unroll n)

LG_HD void p2_full_round(uint32_t s[24], const uint32_t* rk) {
#pragma unroll
  for (int i = 0; i < 24; i++) s[i] = p2_cube(add(s[i], rk[i]));
  p2_external(s);
}

// Pairwise sum of v[0..N): depth log2(N) instead of N - 1.
template <int N> LG_HD uint32_t tree_sum(const uint32_t* v) {
  if constexpr (N == 1) return v[0];
  else return add(tree_sum<N / 2>(v), tree_sum<N - N / 2>(v + N / 2));
}

constexpr uint32_t P2_DIAG_C[24] = LG_P2_DIAG_INIT;
static_assert(P2_DIAG_C[1] == MONT_ONE, "internal diagonal entry 1 is 1");

// The internal diagonal as canonical constants with their Shoup companions
// (products by d_i need no 64-bit multiply).
struct P2DiagShoup { uint32_t w[24], ws[24]; };
constexpr P2DiagShoup make_p2_diag_shoup() {
  P2DiagShoup d{};
  for (int i = 0; i < 24; i++) {
    d.w[i] = cx_from_mont(P2_DIAG_C[i]);
    d.ws[i] = shoup(d.w[i]);
  }
  return d;
}
constexpr P2DiagShoup P2_DSH_H = make_p2_diag_shoup();
static_assert(P2_DSH_H.w[1] == 1, "internal diagonal entry 1 is 1");
static_assert(P2_DSH_H.w[0] == P - 2, "internal diagonal entry 0 is -2: s_0 <- sum + d_0 u = R - u");
constexpr uint32_t C23 = 23, C23_SH = shoup(23);  // the carried sum (p2_coop.cuh)

// Products by +-2^-k (17 of the 24 diagonal entries, and squares of them).  With
// x = hi 2^k + lo (lo < 2^k) and 2^k (p - 1)/2^k = p - 1 = -1 mod p,
//   x 2^-k = hi + lo 2^-k = hi - lo (p - 1)/2^k  (mod p):
// a shift, a mask and one multiply by a small constant in place of Shoup's
// three multiplies.  For x < 2p both hi and lo (p - 1)/2^k are below p, so
// t = +-(hi - lo c) lies in (-p, p) and min(t, t + p) on unsigned words is
// its residue in [0, p).  Montgomery words need no conversion (linear map).
template <int K, bool NEG> LG_HD uint32_t mul_pow2_inv(uint32_t x) {
  static_assert(K >= 1 && K <= 24, "p - 1 = 127 2^24");
  constexpr uint32_t c = (P - 1) >> K;
  const uint32_t lo = x & ((1u << K) - 1), hi = x >> K;
  const uint32_t t = NEG ? lo * c - hi : hi - lo * c;
  return umin(t, t + P);
}
constexpr uint32_t cx_pow2_inv(int k, bool neg) {
  const uint32_t v = cx_pow((P + 1) / 2, (uint64_t)k);
  return neg ? (P - v) % P : v;
}

// Product by the constant W (canonical) with its Shoup companion.
template <uint32_t W> struct P2Shoup { static constexpr uint32_t ws = shoup(W); };
template <uint32_t W> LG_HD uint32_t mul_const(uint32_t x) { return mulc(x, W, P2Shoup<W>::ws); }

// Partial rounds (S-box on lane 0, internal layer 1.1^T + diag).  With
// R = s_1 + ... + s_23 carried from round to round, one round is
//   u = S(s_0 + c),  sum = u + R,  s_0 <- sum + d_0 u = R - u,
//   s_i <- sum + d_i s_i,  R <- 23 sum + D,  D = sum_{i>=1} d_i s_i,
// the same linear map with the products off the S-box's dependent chain.
//
// Eighteen of the 23 diagonal entries come in pairs (d, -d).  For the lanes
// (a, b) of such a pair the half sum S = (a + b)/2 and the half difference
// M = (a - b)/2 follow S <- sum + d M and M <- d S, so
//   S(r + 1) = sum(r) + d^2 S(r - 1),
// and the pair's share of D is 2 d M = 2 d^2 S(r - 1): one product, one
// addition and one summand per pair and round where the two lanes took two of
// each.  S(-1) = M(0)/d starts the recurrence; at the end a = S + M and
// b = S - M with M(r) = d S(r - 1).
//
// S and the five single lanes stay unreduced in [0, 2p) between rounds (their
// only consumer is the next product).  D and 23 sum are summed in 64 bits
// and reduced once: T < 46 p, and with T = h 2^31 + l the value
// l + h (2^24 - 1) = T - h p lies below 2^31 + 46 2^24 < 2p.
//
// What bounds it: the arithmetic pipes (no memory traffic).  2426 warp
// instructions for the 21 rounds against 3636 for the form lane by lane, and
// 25.1 against 38.6 SM clocks per permutation on B200.
constexpr int P2_PAIRS = 9, P2_SINGLES = 5;
// lanes of pair j, its entry d = 2^-k (k > 0) or the integer `num` (k = 0)
struct P2Pair { int a, b, k; uint32_t num; };
constexpr P2Pair p2_pair(int j) {
  return j == 0   ? P2Pair{3, 6, 1, 0}
         : j == 1 ? P2Pair{4, 7, 0, 3}
         : j == 2 ? P2Pair{5, 8, 0, 4}
         : j == 3 ? P2Pair{9, 16, 8, 0}
         : j == 4 ? P2Pair{11, 17, 3, 0}
         : j == 5 ? P2Pair{12, 18, 4, 0}
         : j == 6 ? P2Pair{13, 19, 5, 0}
         : j == 7 ? P2Pair{14, 20, 6, 0}
                  : P2Pair{15, 23, 24, 0};
}
template <int J> struct P2PairC {
  static constexpr int a = p2_pair(J).a, b = p2_pair(J).b, k = p2_pair(J).k;
  static constexpr uint32_t d = k ? cx_pow2_inv(k, false) : p2_pair(J).num;  // canonical
  static constexpr uint32_t d2 = cx_mulmod(d, d);
  static constexpr uint32_t inv_2d = cx_pow(cx_mulmod(2, d), P - 2);
  static_assert(P2_DSH_H.w[a] == d && P2_DSH_H.w[b] == P - d, "the pair's diagonal entries are d and -d");
};
template <int J> LG_HD uint32_t p2_mul_d(uint32_t x) {
  if constexpr (P2PairC<J>::k) return mul_pow2_inv<P2PairC<J>::k, false>(x);
  else return mul_const<P2PairC<J>::d>(x);
}
template <int J> LG_HD uint32_t p2_mul_d2(uint32_t x) {
  constexpr int k2 = 2 * P2PairC<J>::k;
  if constexpr (k2 && k2 <= 24) return mul_pow2_inv<k2, false>(x);
  else return mul_const<P2PairC<J>::d2>(x);
}
template <int J = 0> LG_HD void p2_pairs_in(const uint32_t* s, uint32_t* cur, uint32_t* prev) {
  if constexpr (J < P2_PAIRS) {
    using C = P2PairC<J>;
    const uint32_t a = s[C::a], b = s[C::b];
    cur[J] = mul_pow2_inv<1, false>(a + b);
    if constexpr (C::inv_2d == 1) prev[J] = sub(a, b);
    else prev[J] = mul_const<C::inv_2d>(sub_lazy(a, b));
    p2_pairs_in<J + 1>(s, cur, prev);
  }
}
template <int J = 0> LG_HD void p2_pairs_out(uint32_t* s, const uint32_t* cur, const uint32_t* prev) {
  if constexpr (J < P2_PAIRS) {
    using C = P2PairC<J>;
    const uint32_t c = red(cur[J]), m = p2_mul_d<J>(prev[J]);
    s[C::a] = add(c, m);
    s[C::b] = sub(c, m);
    p2_pairs_out<J + 1>(s, cur, prev);
  }
}
template <int J = 0> LG_HD void p2_pairs_d2(const uint32_t* prev, uint32_t* q) {
  if constexpr (J < P2_PAIRS) {
    q[J] = p2_mul_d2<J>(prev[J]);
    p2_pairs_d2<J + 1>(prev, q);
  }
}
static_assert(P2_DSH_H.w[2] == 2 && P2_DSH_H.w[10] == cx_pow2_inv(2, false) && P2_DSH_H.w[21] == cx_pow2_inv(7, true) &&
                  P2_DSH_H.w[22] == cx_pow2_inv(9, true),
              "the single lanes 2, 10, 21, 22 (lane 1: checked above)");

// One partial round.  x = s_0 + this round's key; `prev` holds S(r - 1) and
// becomes S(r + 1); `single`: the lanes 1, 2, 10, 21, 22.
LG_HD void p2_partial_round(uint32_t* prev, uint32_t* single, uint32_t& x, uint32_t& R, uint32_t key_next) {
  uint32_t q[P2_PAIRS], p[P2_SINGLES];
  p2_pairs_d2(prev, q);
  p[0] = red(single[0]);
  p[1] = dbl(red(single[1]));
  p[2] = mul_pow2_inv<2, false>(single[2]);
  p[3] = mul_pow2_inv<7, true>(single[3]);
  p[4] = mul_pow2_inv<9, true>(single[4]);
  const uint32_t u = p2_cube(x);
  x = sub(add(R, key_next), u);
  const uint32_t sum = add(u, R);
  // two summands in [0, p) fit a word: 64-bit additions of their word sums
  uint64_t A = (uint64_t)(q[0] + q[1]) + (q[2] + q[3]);
  A += q[4] + q[5];
  A += q[6] + q[7];
  A += q[8];
  uint64_t B = (uint64_t)(p[0] + p[1]) + (p[2] + p[3]);
  B += p[4];
  const uint64_t T = A + A + B + (uint64_t)sum * 23u;
  R = red((uint32_t)(T >> 31) * 0x00ffffffu + ((uint32_t)T & 0x7fffffffu));
#pragma unroll
  for (int j = 0; j < P2_PAIRS; j++) prev[j] = sum + q[j];
#pragma unroll
  for (int j = 0; j < P2_SINGLES; j++) single[j] = sum + p[j];
}

LG_HD void p2_partial_rounds(uint32_t s[24]) {
  uint32_t cur[P2_PAIRS], prev[P2_PAIRS], single[P2_SINGLES] = {s[1], s[2], s[10], s[21], s[22]};
  uint32_t R = tree_sum<23>(s + 1);
  p2_pairs_in(s, cur, prev);
  uint32_t x = add(s[0], LG_P2_PARTIAL_RK[0]);
  // two rounds a turn, so that S(r) and S(r - 1) trade places without copies
  LG_UNROLL(1)
  for (int r = 0; r < 20; r += 2) {
    p2_partial_round(prev, single, x, R, LG_P2_PARTIAL_RK[r + 1]);
    p2_partial_round(cur, single, x, R, LG_P2_PARTIAL_RK[r + 2]);
  }
  p2_partial_round(prev, single, x, R, 0);
  s[0] = x;
  p2_pairs_out(s, prev, cur);
  s[1] = red(single[0]);
  s[2] = red(single[1]);
  s[10] = red(single[2]);
  s[21] = red(single[3]);
  s[22] = red(single[4]);
}

LG_HD void p2_permute(uint32_t s[24]) {
  p2_external(s);
  LG_UNROLL(1)
  for (int r = 0; r < 3; r++) p2_full_round(s, LG_P2_FULL_RK[r]);
  p2_partial_rounds(s);
  LG_UNROLL(1)
  for (int r = 3; r < 6; r++) p2_full_round(s, LG_P2_FULL_RK[r]);
}

// node = first 8 lanes of Perm([tag, 0 x7, left, right])
// (internal/hash/poseidon2.go:409-422); tag given in Montgomery form.
LG_HD void p2_compress(uint32_t tag_m, const uint32_t l[8], const uint32_t r[8], uint32_t out[8]) {
  uint32_t s[24];
  s[0] = tag_m;
#pragma unroll
  for (int i = 1; i < 8; i++) s[i] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) { s[8 + i] = l[i]; s[16 + i] = r[i]; }
  p2_permute(s);
#pragma unroll
  for (int i = 0; i < 8; i++) out[i] = s[i];
}

// The host's permutation for the transcript (p2_host.cpp): the same map as
// p2_permute, vectorised when the CPU has AVX2.
void p2_permute_host(uint32_t s[24]);
// The same with a given vector width (2: AVX-512, 1: AVX2, 0: scalar; the
// caller checks the CPU has it) and the width p2_permute_host uses.
void p2_permute_host_at(uint32_t s[24], int level);
int p2_host_simd_level();

// Host sponge: width 24, rate 16, overwrite mode, no padding
// (internal/hash/poseidon2.go:165-255).
struct HostSponge {
  uint32_t state[24];
  uint32_t block[16];
  int len = 0;
  bool wrote = false;
  HostSponge() { reset(); }
  void reset() {
    for (int i = 0; i < 24; i++) state[i] = 0;
    for (int i = 0; i < 16; i++) block[i] = 0;
    len = 0;
    wrote = false;
  }
  void write(uint32_t x_mont) {
    block[len++] = x_mont;
    if (len == 16) {
      for (int i = 0; i < 16; i++) state[i] = block[i];
      p2_permute_host(state);
      for (int i = 0; i < 16; i++) block[i] = 0;
      len = 0;
      wrote = true;
    }
  }
  void sum(uint32_t out[8]) {
    if (!wrote && len == 0) { for (int i = 0; i < 8; i++) out[i] = 0; return; }
    if (len > 0) {
      for (int i = 0; i < len; i++) state[i] = block[i];
      p2_permute_host(state);
      for (int i = 0; i < 16; i++) block[i] = 0;
      len = 0;
      wrote = true;
    }
    for (int i = 0; i < 8; i++) out[i] = state[i];
  }
};

}  // namespace lg
