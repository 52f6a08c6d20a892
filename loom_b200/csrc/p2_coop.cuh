// Cooperative Poseidon2 width 24: six lanes of a warp share one permutation.
// Lane i of a group (i = lane % 6, groups of lanes 0-5, 6-11, ..., 24-29)
// holds state[4i .. 4i+3], one chunk of the external layer's M4 blocks, so
// circ(2 M4, M4, ...) is lane-local except for its four column sums, and the
// internal layer needs one sum over the group.  Both are 3-shuffle
// all-reductions over the six lanes.  Lanes 30 and 31 run the same code on
// dummy data so every shuffle has the full warp.
//
// The form for little parallelism (Merkle tree tops, small trees, the
// transcript): what bounds it is the length of the dependent chain, not the
// instruction count (a warp's permutation is 2,400 instructions in 5,229 cycles).  Round structure as recursion/p2_air.go:206-300.
#pragma once
#include "poseidon2.cuh"

namespace lg {

// The partial rounds' shares of the six lanes: the pairs (d, -d) of
// p2_partial_rounds, two slots a lane (nine of the twelve taken), and the
// single lanes, one slot a lane (five of six).  Per slot the state indices and
// the constants with their Shoup companions; an empty slot has zeros.
struct alignas(16) P2CoopShare {
  uint32_t a[2], b[2], single;             // state indices (24: none)
  uint32_t d2[2], d2s[2], d[2], ds[2];     // pairs: d^2 and d
  uint32_t e[2], es[2];                    // single: d and d^2
  uint32_t pad[3];
};
constexpr P2CoopShare make_p2_coop_share(int lane) {
  constexpr uint32_t singles[5] = {1, 2, 10, 21, 22};
  P2CoopShare c{};
  for (int k = 0; k < 2; k++) {
    c.a[k] = c.b[k] = 24;
    const int j = lane + 6 * k;
    if (j >= P2_PAIRS) continue;
    c.a[k] = (uint32_t)p2_pair(j).a;
    c.b[k] = (uint32_t)p2_pair(j).b;
    c.d[k] = P2_DSH_H.w[c.a[k]];
    c.ds[k] = shoup(c.d[k]);
    c.d2[k] = cx_mulmod(c.d[k], c.d[k]);
    c.d2s[k] = shoup(c.d2[k]);
  }
  c.single = 24;
  if (lane < P2_SINGLES) {
    c.single = singles[lane];
    c.e[0] = P2_DSH_H.w[c.single];
    c.es[0] = shoup(c.e[0]);
    c.e[1] = cx_mulmod(c.e[0], c.e[0]);
    c.es[1] = shoup(c.e[1]);
  }
  return c;
}
// The full-round keys and the lanes' shares, in global memory: blocks copy them
// to shared memory with coalesced loads.  (From constant memory, whose reads by
// lane take a turn per address, they cost each launch about a microsecond.)
struct P2CoopTable {
  uint32_t key[6][24];
  P2CoopShare lane[6];
};
constexpr P2CoopTable make_p2_coop_table() {
  P2CoopTable t{};
  constexpr uint32_t rk[6][24] = LG_P2_FULL_RK_INIT;
  for (int r = 0; r < 6; r++)
    for (int i = 0; i < 24; i++) t.key[r][i] = rk[r][i];
  for (int i = 0; i < 6; i++) t.lane[i] = make_p2_coop_share(i);
  return t;
}
__device__ const P2CoopTable P2_COOP_D = make_p2_coop_table();
constexpr uint32_t P2C_TABLE = sizeof(P2CoopTable) / 4;
constexpr uint32_t p2_single_sum() {
  uint64_t s = 0;
  for (int i : {1, 2, 10, 21, 22}) s += P2_DSH_H.w[i];
  return (uint32_t)(s % P);
}
constexpr uint32_t P2_C1 = p2_single_sum(), P2_C1_SH = shoup(P2_C1);  // the sum of the single lanes' entries

struct P2Lane {
  int lane, base, idx;  // warp lane, first lane of the group, index in the group (0..5)
  P2CoopShare sh;       // this lane's share of the partial rounds
  // `smem`: filled by p2_load_full_keys
  __device__ __forceinline__ void init(const uint32_t* smem) {
    lane = threadIdx.x & 31;
    idx = lane % 6;
    base = lane - idx;
    sh = reinterpret_cast<const P2CoopTable*>(smem)->lane[idx];
  }
  __device__ __forceinline__ int at(int k) const { return (base + ((idx + k) % 6)) & 31; }
  // sum over the group's six lanes, in every lane
  __device__ __forceinline__ uint32_t allreduce(uint32_t v) const {
    uint32_t s1 = add(v, __shfl_sync(0xffffffffu, v, (base + (idx ^ 1)) & 31));
    uint32_t s2 = add(s1, __shfl_sync(0xffffffffu, s1, at(2)));
    return add(s2, __shfl_sync(0xffffffffu, s1, at(4)));
  }
};

// Shared memory of a block that runs cooperative permutations: the table above
// (the keys first), then per warp six groups' states (five and the dummy), through which
// the lanes trade their chunks for the partial rounds' shares and back (25
// words a group: the last one takes the empty slots' writes).
constexpr uint32_t P2C_GROUP = 28;  // words per group, a multiple of four
LG_HD constexpr uint32_t p2c_smem_words(uint32_t warps) { return P2C_TABLE + warps * 6 * P2C_GROUP; }
__device__ __forceinline__ void p2_load_full_keys(uint32_t* smem) {
  for (uint32_t i = threadIdx.x; i < P2C_TABLE; i += blockDim.x) smem[i] = __ldg(reinterpret_cast<const uint32_t*>(&P2_COOP_D) + i);
  __syncthreads();
}

__device__ __forceinline__ void p2c_external(uint32_t x[4], const P2Lane& L) {
  p2_m4(x[0], x[1], x[2], x[3]);
  uint32_t c0 = L.allreduce(x[0]), c1 = L.allreduce(x[1]), c2 = L.allreduce(x[2]), c3 = L.allreduce(x[3]);
  x[0] = add(x[0], c0);
  x[1] = add(x[1], c1);
  x[2] = add(x[2], c2);
  x[3] = add(x[3], c3);
}

__device__ __forceinline__ void p2c_full(uint32_t x[4], const P2Lane& L, const uint32_t* keys /*24 words*/) {
#pragma unroll
  for (int i = 0; i < 4; i++) x[i] = p2_cube(add(x[i], keys[4 * L.idx + i]));
  p2c_external(x, L);
}

// The partial rounds in the pair form of p2_partial_rounds, with S = a + b
// (not halved: S <- 2 sum + d M) and every lane of the group carrying its own
// copy of s_0 and R.  D(r), the group's sum, would wait for the single lanes'
// values of the same round; with
//   sum_i d_i s_i(r) = c1 sum(r - 1) + sum_i d_i^2 s_i(r - 1)
// (c1: the sum of their d_i) everything that crosses lanes is known a round
// earlier, so the all-reduction for round r + 1 runs beside round r's S-box
// and the dependent chain of a round is the S-box and one subtraction.
__device__ __forceinline__ void p2c_partial(uint32_t x[4], const P2Lane& L, uint32_t* st /*the group's words*/) {
  const P2CoopShare& c = L.sh;
  *reinterpret_cast<uint4*>(st + 4 * L.idx) = make_uint4(x[0], x[1], x[2], x[3]);
  __syncwarp();
  uint32_t R = L.allreduce(add(add(L.idx ? x[0] : 0u, x[1]), add(x[2], x[3])));
  // per slot S(r), S(r - 1) (for the way out), q(r) = d^2 S(r - 1) = d M(r) and
  // q(r - 1) (f0, f1); for the single s(r) and p = d s(r).  Round r's values
  // come from sum(r - 1) and the round before's products.
  uint32_t S0, S1, s, P0 = 0, P1 = 0, q0, q1, f0 = 0, f1 = 0, p;
  {
    const uint32_t a0 = st[c.a[0]], b0 = st[c.b[0]], a1 = st[c.a[1]], b1 = st[c.b[1]];
    s = st[c.single];
    S0 = a0 + b0;
    S1 = a1 + b1;
    q0 = mulc(sub_lazy(a0, b0), c.d[0], c.ds[0]);
    q1 = mulc(sub_lazy(a1, b1), c.d[1], c.ds[1]);
    p = mulc(s, c.e[0], c.es[0]);
  }
  uint32_t X = add(st[0], P2_PARTIAL_RK_D[0]), Rk = add(R, P2_PARTIAL_RK_D[1]);
  uint32_t t = add(add(q0, q1), p), k1 = 0, sum = 0;
#pragma unroll 3
  for (int r = 0; r < 21; r++) {
    const uint32_t ta = __shfl_sync(0xffffffffu, t, (L.base + (L.idx ^ 1)) & 31);
    const uint32_t y = mul_lazy(X, X);
    if (r) {  // the state before this round, from the last one's sum
      const uint32_t sum2 = dbl(sum);
      S0 = sum2 + f0;
      S1 = sum2 + f1;
      s = sum + p;
    }
    const uint32_t n0 = mulc(S0, c.d2[0], c.d2s[0]), n1 = mulc(S1, c.d2[1], c.d2s[1]);
    const uint32_t e = mulc(s, c.e[1], c.es[1]);
    const uint32_t t1 = add(t, ta);
    const uint32_t tb = __shfl_sync(0xffffffffu, t1, L.at(2)), tc = __shfl_sync(0xffffffffu, t1, L.at(4));
    const uint32_t u = mul(y, X);
    if (r) p = mulc(s, c.e[0], c.es[0]);
    X = sub(Rk, u);
    sum = add(u, R);
    t = add(add(n0, n1), e);
    const uint32_t A = add(add(k1, t1), add(tb, tc));
    k1 = mulc(sum, P2_C1, P2_C1_SH);
    R = add(mulc(sum, C23, C23_SH), A);
    Rk = add(R, r < 19 ? P2_PARTIAL_RK_D[r < 19 ? r + 2 : 0] : 0u);
    P0 = S0;
    P1 = S1;
    f0 = q0;
    f1 = q1;
    q0 = n0;
    q1 = n1;
  }
  {
    const uint32_t sum2 = dbl(sum);
    S0 = sum2 + f0;
    S1 = sum2 + f1;
    s = sum + p;
  }
  const uint32_t m0 = mulc(P0, c.d[0], c.ds[0]), m1 = mulc(P1, c.d[1], c.ds[1]);
  S0 = red(S0);
  S1 = red(S1);
  __syncwarp();
  st[c.a[0]] = mul_pow2_inv<1, false>(S0 + m0);
  st[c.b[0]] = mul_pow2_inv<1, false>(sub_lazy(S0, m0));
  st[c.a[1]] = mul_pow2_inv<1, false>(S1 + m1);
  st[c.b[1]] = mul_pow2_inv<1, false>(sub_lazy(S1, m1));
  st[c.single] = red(s);
  if (L.idx == 0) st[0] = X;
  __syncwarp();
  const uint4 v = *reinterpret_cast<const uint4*>(st + 4 * L.idx);
  x[0] = v.x;
  x[1] = v.y;
  x[2] = v.z;
  x[3] = v.w;
  __syncwarp();
}

// smem: the block's p2c_smem_words.
__device__ __forceinline__ void p2c_permute(uint32_t x[4], const P2Lane& L, uint32_t* smem) {
  p2c_external(x, L);
#pragma unroll 1
  for (int r = 0; r < 3; r++) p2c_full(x, L, smem + 24 * r);
  p2c_partial(x, L, smem + P2C_TABLE + ((threadIdx.x >> 5) * 6 + (uint32_t)L.base / 6) * P2C_GROUP);
#pragma unroll 1
  for (int r = 3; r < 6; r++) p2c_full(x, L, smem + 24 * r);
}
// Node compression H(left, right) with the digests held as: left in lanes
// idx 2, 3 and right in lanes idx 4, 5 (4 words each); the result lands in
// lanes idx 0, 1.
__device__ __forceinline__ void p2c_compress(uint32_t x[4], const P2Lane& L, uint32_t* smem) {
  if (L.idx == 0) { x[0] = to_mont(0x4e4f4445u); x[1] = x[2] = x[3] = 0; }
  if (L.idx == 1) { x[0] = x[1] = x[2] = x[3] = 0; }
  p2c_permute(x, L, smem);
}

// Moves a digest from lanes idx 0, 1 to lanes idx 2, 3 (the left input slot).
__device__ __forceinline__ void p2c_digest_to_left(uint32_t x[4], const P2Lane& L) {
  uint32_t y[4];
#pragma unroll
  for (int i = 0; i < 4; i++) y[i] = __shfl_sync(0xffffffffu, x[i], (L.base + ((L.idx + 4) % 6)) & 31);
  if (L.idx == 2 || L.idx == 3)
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = y[i];
}

}  // namespace lg
