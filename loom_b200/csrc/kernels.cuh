// sm_100a kernels of the Poseidon2 prove path.  All field data is Montgomery
// words; an E6 column is stored as 6 base "lanes" (structure of arrays), so
// every transform and gather works on plain u32 columns.
#pragma once
#include <cuda_runtime.h>

#include "field.cuh"
#include "p2_coop.cuh"
#include "ntt16.cuh"
#include "scan.cuh"

namespace lg {

constexpr int RATE_LOG = 2;  // blowup 4 (internal/constants/const.go:24)
constexpr int SMEM_NTT_MAX_LOG = 14;
constexpr uint32_t LEAF_TAG = 0x4c454146u, NODE_TAG = 0x4e4f4445u;

// ---------------------------------------------------------------- twiddles
// tw[j] = w_n^j for j < n, w_n = root_of_unity(log n).
__global__ void k_fill_powers(uint32_t* out, uint64_t n, uint32_t base, uint32_t start) {
  uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (j < n) out[j] = mul(start, mont_pow(base, j));
}

// tau[B] = w^bitrev_logm(B) for B < 2^logm, w of order 2^(logm + 1): canonical
// words with their Shoup companions (the forward tree, ntt_large.cuh).
__global__ void k_fill_tree(uint2* out, int logm, uint32_t w) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >> logm) return;
  const uint32_t c = from_mont(mont_pow(w, bitrev32(b, logm)));
  out[b] = make_uint2(c, (uint32_t)(((uint64_t)c << 32) / P));
}

// ---------------------------------------------------------------- smem NTT
// Radix-2 stages over a block-resident array A of n = 2^logn words.
// tw: table of w_n^j (j < n) for this n; `inverse` uses w_n^-j = w_n^(n-j).
__device__ __forceinline__ uint32_t tw_at(const uint32_t* tw, uint32_t idx, uint32_t mask, bool inverse) {
  return inverse ? __ldg(tw + ((0u - idx) & mask)) : __ldg(tw + idx);
}

// DIT: bit-reversed input, natural output.
__device__ void smem_dit(uint32_t* A, int logn, const uint32_t* tw, bool inverse) {
  const uint32_t n = 1u << logn, mask = n - 1;
  for (int s = 1; s <= logn; s++) {
    const uint32_t half = 1u << (s - 1);
    for (uint32_t t = threadIdx.x; t < n / 2; t += blockDim.x) {
      uint32_t j = t & (half - 1);
      uint32_t i0 = ((t >> (s - 1)) << s) | j, i1 = i0 + half;
      uint32_t w = tw_at(tw, j << (logn - s), mask, inverse);
      uint32_t u = A[i0], v = mul(A[i1], w);
      A[i0] = add(u, v);
      A[i1] = sub(u, v);
    }
    __syncthreads();
  }
}

// DIF: natural input, bit-reversed output.
__device__ void smem_dif(uint32_t* A, int logn, const uint32_t* tw, bool inverse) {
  const uint32_t n = 1u << logn, mask = n - 1;
  for (int s = logn; s >= 1; s--) {
    const uint32_t half = 1u << (s - 1);
    for (uint32_t t = threadIdx.x; t < n / 2; t += blockDim.x) {
      uint32_t j = t & (half - 1);
      uint32_t i0 = ((t >> (s - 1)) << s) | j, i1 = i0 + half;
      uint32_t w = tw_at(tw, j << (logn - s), mask, inverse);
      uint32_t u = A[i0], v = A[i1];
      A[i0] = add(u, v);
      A[i1] = mul(sub_lazy(u, v), w);
    }
    __syncthreads();
  }
}

// Inverse transform of natural-order values to natural-order coefficients
// (scaled by 1/n), in place; one block per lane, lanes[blockIdx.x].
// n >= 16: DIT whose first pass gathers the bit-reversed input from global
// memory; smaller n: radix-2 stages in shared memory.
// LOGN: the size when fixed at compile time (2^4..2^14), else 0 and logn_rt.
template <int LOGN>
__global__ void k_intt(uint32_t* const* lanes, int logn_rt, const uint32_t* tw_n, uint32_t n_inv) {
  const int logn = LOGN ? LOGN : logn_rt;
  extern __shared__ uint32_t sm[];
  const uint32_t n = 1u << logn;
  uint32_t* d = lanes[blockIdx.x];
  if (logn < 4) {
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) sm[bitrev32(k, logn)] = d[k];
    __syncthreads();
    smem_dit(sm, logn, tw_n, true);
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) d[k] = mul(sm[k], n_inv);
    return;
  }
  auto first = [&](uint32_t t, uint32_t r, int lo) { return d[bitrev32(grp_index(t, r, lo), logn)]; };
  auto store = [&](uint32_t t, int lo, const uint32_t* v) {
#pragma unroll
    for (uint32_t r = 0; r < 16; r++) d[grp_index(t, r, lo)] = mul(v[r], n_inv);
  };
  ntt16<false>(sm, logn, tw_n, true, first, store);
}

// LDE of one lane per block: Lagrange values in natural order (or canonical
// coefficients when from_coeffs) -> for coset a < 4,
// out[a n + b] = P(w_4n^bitrev2(a) w_n^bitrev(b)), the bit-reversed
// evaluations on <w_4n> of reedsolomon.Encode (internal/reedsolomon/rs.go:52-70).
// Optionally writes the coefficients.  Shared memory: A (coefficients) and B
// (work), pad16 layout.
// 4-byte asynchronous copy global -> shared (cp.async, no register staging):
// a thread issues all of its copies before waiting for any.
__device__ __forceinline__ void cp_async4(uint32_t* smem, const uint32_t* gmem) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

struct LdeLane { const uint32_t* src; uint32_t* out; uint32_t* coef; };
// fwd = 0: only the inverse transform, coset 0 and the coefficients (L.coef,
// which must be set); k_lde_fwd then runs the other cosets.
template <int LOGN>
__global__ void k_lde(const LdeLane* lanes, int logn_rt, int from_coeffs, const uint32_t* tw_n, const uint32_t* tw_4n,
                      uint32_t n_inv, int fwd = 1) {
  const int logn = LOGN ? LOGN : logn_rt;
  extern __shared__ uint32_t sm[];
  const uint32_t n = 1u << logn;
  const LdeLane L = lanes[blockIdx.x];
  const uint32_t big = n << RATE_LOG;
  if (logn < 4) {  // tiny columns: radix-2 stages
    uint32_t* A = sm;
    uint32_t* B = sm + n;
    if (from_coeffs) {
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) A[k] = L.src[k];
      __syncthreads();
    } else {
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) A[bitrev32(k, logn)] = L.src[k];
      __syncthreads();
      smem_dit(A, logn, tw_n, true);
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) A[k] = mul(A[k], n_inv);
      __syncthreads();
    }
    if (L.coef)
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) L.coef[k] = A[k];
    for (int a = 0; a < (1 << RATE_LOG); a++) {
      const uint32_t e = bitrev32((uint32_t)a, RATE_LOG);
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) B[k] = mul(A[k], __ldg(tw_4n + ((e * k) & (big - 1))));
      __syncthreads();
      smem_dif(B, logn, tw_n, false);
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) L.out[(uint64_t)a * n + k] = B[k];
      __syncthreads();
    }
    return;
  }
  uint32_t* A = sm;
  uint32_t* B = sm + pad16(n);
  if (from_coeffs) {
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
      uint32_t v = L.src[k];
      A[pad16(k)] = v;
      if (L.coef) L.coef[k] = v;
    }
    __syncthreads();
  } else {
    // the input goes to B (free until the coset transforms) with coalesced
    // loads; the first pass gathers it in bit-reversed order from there
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) B[pad16(k)] = L.src[k];
    __syncthreads();
    auto first = [&](uint32_t t, uint32_t r, int lo) { return B[pad16(bitrev32(grp_index(t, r, lo), logn))]; };
    auto store = [&](uint32_t t, int lo, const uint32_t* v) {
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        uint32_t i = grp_index(t, r, lo), c = mul(v[r], n_inv);
        A[pad16(i)] = c;
        if (L.coef) L.coef[i] = c;
      }
    };
    // Coset 0 is <w_n> itself: its bit-reversed evaluations are the input
    // values in bit-reversed order, which the DIT's first pass (local bits
    // [0, 4): 16 consecutive positions) has just gathered.
    auto coset0 = [&](uint32_t t, const uint32_t* v) {
      uint4* q = reinterpret_cast<uint4*>(L.out + ((uint64_t)t << 4));
      q[0] = make_uint4(v[0], v[1], v[2], v[3]);
      q[1] = make_uint4(v[4], v[5], v[6], v[7]);
      q[2] = make_uint4(v[8], v[9], v[10], v[11]);
      q[3] = make_uint4(v[12], v[13], v[14], v[15]);
    };
    ntt16<false>(A, logn, tw_n, true, first, store, coset0);  // A is both work and result
  }
  if (!fwd) return;
  for (int a = from_coeffs ? 0 : 1; a < (1 << RATE_LOG); a++) {
    const uint32_t e = bitrev32((uint32_t)a, RATE_LOG);
    uint32_t* o = L.out + (uint64_t)a * n;
    auto first = [&](uint32_t t, uint32_t r, int lo) {
      uint32_t i = grp_index(t, r, lo);
      return mul(A[pad16(i)], __ldg(tw_4n + ((e * i) & (big - 1))));
    };
    auto store = [&](uint32_t t, int lo, const uint32_t* v) {
      // DIF's last pass has lo = 0: the group is 16 consecutive outputs
      uint4* q = reinterpret_cast<uint4*>(o + ((uint64_t)t << 4));
      q[0] = make_uint4(v[0], v[1], v[2], v[3]);
      q[1] = make_uint4(v[4], v[5], v[6], v[7]);
      q[2] = make_uint4(v[8], v[9], v[10], v[11]);
      q[3] = make_uint4(v[12], v[13], v[14], v[15]);
    };
    ntt16<true>(B, logn, tw_n, false, first, store);
  }
}

// The coset transforms of the LDE as blocks of their own: block (x, y) runs
// coset a = first + x of lane lane0 + y (the cosets of a lane side by side,
// so its coefficients come from DRAM once and from L2 after) from its
// coefficients (L.coef, or L.src when
// the lane is given as coefficients), written bit-reversed as in k_lde.  One
// shared-memory array per block (the coefficients are read from global
// memory, where the inverse transform left them, rather than kept in shared
// memory), so several blocks share an SM and overlap one another's barriers
// and shared-memory round trips.  MAXT: the block size the kernel is built
// for (registers capped so that 1024 / MAXT blocks fit: 32 warps per SM
// without spills).
// The coset shifts of the first DIF pass: its element i = r 2^(logn-4) + t
// (t < 2^(logn-4)) takes w_4n^(e i) = w_4n^(e t) w_64^(e r), since
// w_4n^(2^(logn-4)) = w_64 for every size; w_64^(e r) for e < 4, r < 16 as
// canonical words with their Shoup companions.
struct CosetSteps { uint32_t w[4][16], ws[4][16]; };
constexpr CosetSteps make_coset_steps() {
  CosetSteps c{};
  for (uint32_t e = 0; e < 4; e++)
    for (uint32_t r = 0; r < 16; r++) {
      c.w[e][r] = cx_pow(3, (uint64_t)((P - 1) / 64) * ((e * r) % 64));
      c.ws[e][r] = shoup(c.w[e][r]);
    }
  return c;
}
__constant__ CosetSteps COSET_STEPS_D = make_coset_steps();

template <int LOGN, int MAXT>
__global__ void __launch_bounds__(MAXT, 1024 / MAXT)
    k_lde_fwd(const LdeLane* lanes, uint32_t lane0, int first, const uint32_t* tw_n, const uint32_t* tw_4n) {
  static_assert(LOGN >= 4, "radix-16 passes");
  extern __shared__ uint32_t sm[];
  constexpr uint32_t n = 1u << LOGN, big = n << RATE_LOG;
  const LdeLane L = lanes[lane0 + blockIdx.y];
  const uint32_t a = first + blockIdx.x;
  const uint32_t e = bitrev32(a, RATE_LOG);
  const uint32_t* coef = L.coef ? L.coef : L.src;
  uint32_t* o = L.out + (uint64_t)a * n;
  // the coefficients go to shared memory first (cp.async, coalesced, all in
  // flight at once); the first pass reads and overwrites its own positions
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) cp_async4(&sm[pad16(k)], coef + k);
  cp_async_wait_all();
  __syncthreads();
  // one table load per group for w_4n^(e t); the 15 other shifts of the group
  // are Shoup products by constants (r is a compile-time index after unrolling)
  uint32_t shift_t = 0;
  auto first_pass = [&](uint32_t t, uint32_t r, int lo) {
    const uint32_t i = grp_index(t, r, lo);
    if (r == 0) shift_t = __ldg(tw_4n + ((e * t) & (big - 1)));
    const uint32_t x = mul(sm[pad16(i)], shift_t);
    return r ? mulc(x, COSET_STEPS_D.w[e][r], COSET_STEPS_D.ws[e][r]) : x;
  };
  auto store = [&](uint32_t t, int lo, const uint32_t* v) {
    uint4* q = reinterpret_cast<uint4*>(o + ((uint64_t)t << 4));
    q[0] = make_uint4(v[0], v[1], v[2], v[3]);
    q[1] = make_uint4(v[4], v[5], v[6], v[7]);
    q[2] = make_uint4(v[8], v[9], v[10], v[11]);
    q[3] = make_uint4(v[12], v[13], v[14], v[15]);
  };
  ntt16<true>(sm, LOGN, tw_n, false, first_pass, store);
}

// The inverse transform of the split LDE, one lane per block with a single
// shared-memory array: the first pass gathers its bit-reversed inputs from
// global memory (the lane's few tens of KB stay in L1 while the block reads
// them), writes coset 0 (the input in bit-reversed order) from those
// registers, and the last pass writes the coefficients to global memory,
// where k_lde_fwd reads them.
template <int LOGN, int MAXT>
__global__ void __launch_bounds__(MAXT, 1024 / MAXT)
    k_lde_inv(const LdeLane* lanes, const uint32_t* tw_n, uint32_t n_inv) {
  static_assert(LOGN >= 4, "radix-16 passes");
  extern __shared__ uint32_t sm[];
  const LdeLane L = lanes[blockIdx.x];
  auto first = [&](uint32_t t, uint32_t r, int lo) { return __ldg(L.src + bitrev32(grp_index(t, r, lo), LOGN)); };
  auto coset0 = [&](uint32_t t, const uint32_t* v) {
    uint4* q = reinterpret_cast<uint4*>(L.out + ((uint64_t)t << 4));
    q[0] = make_uint4(v[0], v[1], v[2], v[3]);
    q[1] = make_uint4(v[4], v[5], v[6], v[7]);
    q[2] = make_uint4(v[8], v[9], v[10], v[11]);
    q[3] = make_uint4(v[12], v[13], v[14], v[15]);
  };
  auto store = [&](uint32_t t, int lo, const uint32_t* v) {
#pragma unroll
    for (uint32_t r = 0; r < 16; r++) L.coef[grp_index(t, r, lo)] = mul(v[r], n_inv);
  };
  ntt16<false>(sm, LOGN, tw_n, true, first, store, coset0);
}

// Evaluations of a coefficient lane on the cosets s_c <w_n>, s_c = g w_4n^c,
// c = blockIdx.y < 4, in natural order: out[c n + j] = P(s_c w_n^j).
// n >= 16: the scaled coefficients coef[k] s_c^k (shift: the table of s_c^k,
// coset_shifts) go to the second half of shared memory with coalesced loads;
// a DIT whose first pass gathers them in bit-reversed order from there works
// in the first half.
struct CosetLane { const uint32_t* src; uint32_t* out; };
template <int LOGN>
__global__ void k_coset_eval(const CosetLane* lanes, int logn_rt, const uint32_t* tw_n, const uint32_t* shift) {
  const int logn = LOGN ? LOGN : logn_rt;
  extern __shared__ uint32_t sm[];
  const uint32_t n = 1u << logn, c = blockIdx.y;
  const CosetLane L = lanes[blockIdx.x];
  const uint32_t* sh = shift + (uint64_t)c * n;
  uint32_t* o = L.out + (uint64_t)c * n;
  if (logn < 4) {
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) sm[k] = mul(L.src[k], sh[k]);
    __syncthreads();
    smem_dif(sm, logn, tw_n, false);
    for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) o[j] = sm[bitrev32(j, logn)];
    return;
  }
  // the coefficients (to S2) and the shift powers (to the work half, free
  // until the first pass) arrive by cp.async, all copies in flight at once;
  // then each thread scales its own words
  uint32_t* S2 = sm + pad16(n) + 1;
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    cp_async4(&S2[pad16(k)], L.src + k);
    cp_async4(&sm[pad16(k)], sh + k);
  }
  cp_async_wait_all();
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) S2[pad16(k)] = mul(S2[pad16(k)], sm[pad16(k)]);
  __syncthreads();
  auto first = [&](uint32_t t, uint32_t r, int lo) { return S2[pad16(bitrev32(grp_index(t, r, lo), logn))]; };
  auto store = [&](uint32_t t, int lo, const uint32_t* v) {
#pragma unroll
    for (uint32_t r = 0; r < 16; r++) o[grp_index(t, r, lo)] = v[r];
  };
  ntt16<false>(sm, logn, tw_n, false, first, store);
}

// ---------------------------------------------------------------- leaves
// leaf k = Sponge(LEAF, 2nB, 2nE, lo.base, hi.base, lo.ext, hi.ext) over
// rows 2k, 2k+1 (internal/fri/hash.go:39-57).  Base lanes at base + c*stride,
// ext column e lane l at ext + (6e + l)*stride.
struct LeafGroup {
  const uint32_t* base;
  const uint32_t* ext;
  uint64_t stride;      // words between lanes
  uint32_t nb, ne;
  uint32_t n_leaves;    // rows / 2
  uint32_t* out;        // n_leaves digests of 8 words
};

__device__ __forceinline__ uint32_t leaf_elem(const LeafGroup& g, uint32_t idx, uint32_t k, uint32_t hdr0,
                                              uint32_t hdr1, uint32_t hdr2) {
  if (idx == 0) return hdr0;
  if (idx == 1) return hdr1;
  if (idx == 2) return hdr2;
  idx -= 3;
  if (idx < 2 * g.nb) {
    uint32_t h = idx >= g.nb;
    uint32_t c = idx - h * g.nb;
    return g.base[c * g.stride + 2 * k + h];
  }
  idx -= 2 * g.nb;
  uint32_t h = idx >= 6 * g.ne;
  uint32_t e = idx - h * 6 * g.ne;
  return g.ext[e * g.stride + 2 * k + h];
}

// Kernels with a permutation per thread: built for blocks of at most 256
// threads and 128 registers, since the permutation keeps its 24 words and the
// products in flight in registers.  With a cap of 64 registers (1024-thread
// blocks) the full rounds take 6.9 SM clocks instead of 6.4 (B200); room for
// more than 128 (blocks of 128, four on an SM) changes nothing.
constexpr int P2_MAX_BLOCK = 256;

// One thread per leaf: the fewest instructions per permutation, for launches
// with enough leaves to fill the GPU.
__global__ void __launch_bounds__(P2_MAX_BLOCK, 2) k_hash_leaves1(const LeafGroup* groups) {
  const LeafGroup g = groups[blockIdx.y];
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g.n_leaves) return;
  const uint32_t total = 3 + 2 * g.nb + 12 * g.ne;
  const uint32_t h0 = to_mont(LEAF_TAG), h1 = to_mont(2 * g.nb), h2 = to_mont(2 * g.ne);
  uint32_t s[24];
#pragma unroll
  for (int i = 0; i < 24; i++) s[i] = 0;
  for (uint32_t b = 0; b < total; b += 16) {
#pragma unroll
    for (uint32_t i = 0; i < 16; i++)
      if (b + i < total) s[i] = leaf_elem(g, b + i, k, h0, h1, h2);
    p2_permute(s);
  }
  uint32_t* o = g.out + (uint64_t)k * 8;
#pragma unroll
  for (int i = 0; i < 8; i++) o[i] = s[i];
}

// Cooperative form: six lanes per leaf (p2_coop.cuh), five leaves per warp.
constexpr uint32_t P2_GROUPS_PER_WARP = 5;

__global__ void k_hash_leaves(const LeafGroup* groups) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(4)];
  p2_load_full_keys(keys);
  P2Lane L;
  L.init(keys);
  const LeafGroup g = groups[blockIdx.y];
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t k = (blockIdx.x * warps + warp) * P2_GROUPS_PER_WARP + (uint32_t)L.base / 6;
  const bool active = L.lane < 30 && k < g.n_leaves;
  const uint32_t total = 3 + 2 * g.nb + 12 * g.ne;
  const uint32_t h0 = to_mont(LEAF_TAG), h1 = to_mont(2 * g.nb), h2 = to_mont(2 * g.ne);
  uint32_t x[4] = {0, 0, 0, 0};
  for (uint32_t b = 0; b < total; b += 16) {
    if (active && L.idx < 4) {
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        uint32_t e = b + 4 * L.idx + i;
        if (e < total) x[i] = leaf_elem(g, e, k, h0, h1, h2);
      }
    }
    p2c_permute(x, L, keys);
  }
  if (active && L.idx < 2) {
    uint32_t* o = g.out + (uint64_t)k * 8 + 4 * L.idx;
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = x[i];
  }
}

// ---------------------------------------------------------------- Merkle
// nodes: 1-indexed, 8 words per node.  Level step: node i = H(2i, 2i+1) for
// i in [start, 2 start); injection fold: node start+j = H(node, inj[j]),
// several injections of the same width chained in schedule order
// (internal/merkle/tree.go:210-327).  Six lanes per node.

// Loads digest words into the left (idx 2, 3) or right (idx 4, 5) slot.
__device__ __forceinline__ void p2c_load_slot(uint32_t x[4], const P2Lane& L, int slot, const uint32_t* digest,
                                              bool active) {
  if (active && (L.idx >> 1) == slot) {
    const uint32_t* d = digest + 4 * (L.idx & 1);
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = d[i];
  }
}
__device__ __forceinline__ void p2c_store_digest(const uint32_t x[4], const P2Lane& L, uint32_t* digest, bool active) {
  if (active && L.idx < 2) {
    uint32_t* d = digest + 4 * L.idx;
#pragma unroll
    for (int i = 0; i < 4; i++) d[i] = x[i];
  }
}

__device__ __forceinline__ void merkle_node(uint32_t* nodes, uint64_t id, const P2Lane& L, uint32_t* keys,
                                            bool active) {
  uint32_t x[4] = {0, 0, 0, 0};
  p2c_load_slot(x, L, 1, nodes + 2 * id * 8, active);
  p2c_load_slot(x, L, 2, nodes + (2 * id + 1) * 8, active);
  p2c_compress(x, L, keys);
  p2c_store_digest(x, L, nodes + id * 8, active);
}

// node = H(... H(H(node, inj_0[j]), inj_1[j]) ..., inj_{n-1}[j])
__device__ __forceinline__ void merkle_chain(uint32_t* nodes, uint64_t id, uint32_t j, const uint32_t* const* inj,
                                             uint32_t n_inj, const P2Lane& L, uint32_t* keys, bool active) {
  if (n_inj == 0) return;
  uint32_t x[4] = {0, 0, 0, 0}, next[4] = {0, 0, 0, 0};
  p2c_load_slot(x, L, 1, nodes + id * 8, active);
  p2c_load_slot(next, L, 2, inj[0] + (uint64_t)j * 8, active);
  for (uint32_t t = 0; t < n_inj; t++) {
    if ((L.idx >> 1) == 2)
#pragma unroll
      for (int i = 0; i < 4; i++) x[i] = next[i];
    if (t + 1 < n_inj) p2c_load_slot(next, L, 2, inj[t + 1] + (uint64_t)j * 8, active);  // beside the permutation
    p2c_compress(x, L, keys);
    if (t + 1 < n_inj) p2c_digest_to_left(x, L);
  }
  p2c_store_digest(x, L, nodes + id * 8, active);
}

__global__ void k_merkle_level(uint32_t* nodes, uint32_t start) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(4)];
  p2_load_full_keys(keys);
  P2Lane L;
  L.init(keys);
  const uint32_t warps = blockDim.x >> 5;
  const uint32_t i = (blockIdx.x * warps + (threadIdx.x >> 5)) * P2_GROUPS_PER_WARP + (uint32_t)L.base / 6;
  merkle_node(nodes, (uint64_t)start + i, L, keys, L.lane < 30 && i < start);
}

__global__ void k_merkle_inject(uint32_t* nodes, uint32_t start, const uint32_t* const* inj, uint32_t n_inj) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(4)];
  p2_load_full_keys(keys);
  P2Lane L;
  L.init(keys);
  const uint32_t warps = blockDim.x >> 5;
  const uint32_t j = (blockIdx.x * warps + (threadIdx.x >> 5)) * P2_GROUPS_PER_WARP + (uint32_t)L.base / 6;
  merkle_chain(nodes, (uint64_t)start + j, j, inj, n_inj, L, keys, L.lane < 30 && j < start);
}

// One thread per node (levels and injection chains wide enough to fill the
// GPU): the fewest instructions per permutation.  Digests are 32-byte
// aligned, so they move as two 16-byte words.
__device__ __forceinline__ void ld_digest(const uint32_t* p, uint32_t d[8]) {
  const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
  d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}
__device__ __forceinline__ void st_digest(uint32_t* p, const uint32_t d[8]) {
  reinterpret_cast<uint4*>(p)[0] = make_uint4(d[0], d[1], d[2], d[3]);
  reinterpret_cast<uint4*>(p)[1] = make_uint4(d[4], d[5], d[6], d[7]);
}
__global__ void __launch_bounds__(P2_MAX_BLOCK, 2) k_merkle_level1(uint32_t* nodes, uint32_t start) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= start) return;
  const uint64_t id = (uint64_t)start + i;
  uint32_t l[8], r[8];
  ld_digest(nodes + 2 * id * 8, l);
  ld_digest(nodes + (2 * id + 1) * 8, r);
  p2_compress(to_mont(NODE_TAG), l, r, l);
  st_digest(nodes + id * 8, l);
}
__global__ void __launch_bounds__(P2_MAX_BLOCK, 2) k_merkle_inject1(uint32_t* nodes, uint32_t start, const uint32_t* const* inj, uint32_t n_inj) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= start) return;
  uint32_t* nd = nodes + ((uint64_t)start + j) * 8;
  uint32_t l[8], r[8], next[8];
  ld_digest(nd, l);
  ld_digest(inj[0] + (uint64_t)j * 8, next);
  for (uint32_t t = 0; t < n_inj; t++) {
#pragma unroll
    for (int w = 0; w < 8; w++) r[w] = next[w];
    if (t + 1 < n_inj) ld_digest(inj[t + 1] + (uint64_t)j * 8, next);  // beside the permutation
    p2_compress(to_mont(NODE_TAG), l, r, l);
  }
  st_digest(nd, l);
}

// Upper tree levels, one subtree per block: block b of B (gridDim.x) owns the
// nodes [b top/B, (b+1) top/B) of width `top` and, for each width w from
// top/2 down to B, runs the 2-to-1 step over its share of the level, then the
// injections of width w in schedule order, with a block barrier between
// levels.  One block (B = 1) builds a whole tree top; B > 1 replaces the
// launches of the levels top/2 .. B, which are latency bound, by one.  When
// fold_first, the injections of width `top` fold first (a tree whose leaf
// level fits in one block).
// With fs.out set (one block only), the block then hashes the challenge that
// binds the root: fs.out = sponge(fs.pre[0..n_pre) || fs.prev[0..8) || root),
// as k_fs_challenge, which it replaces for the FRI layer trees.
struct InjRef { const uint32_t* leaves; uint32_t width; };
struct FsTail { const uint32_t* pre; uint32_t n_pre; const uint32_t* prev; uint32_t* out; };
// A block of 1024 threads would leave each 64 registers, which is just what the
// kernel takes (71 when nvcc compiles the unit in parts, and such a block does
// not start); blocks have at most 512, with room for twice as many, and the
// widest levels take more turns.  Not a launch bound: compiled for one, the
// kernel has the same registers and is 1-4 us slower a tree of 2^11 or 2^13
// leaves (B200: 84 -> 88 and 96 -> 97 us).
constexpr int MERKLE_TAIL_BLOCK = 512;
__global__ void k_merkle_tail(uint32_t* nodes, uint32_t top, int fold_first, const InjRef* inj, uint32_t n_inj,
                              FsTail fs) {
  extern __shared__ __align__(16) uint32_t keys[];  // p2c_smem_words(warps)
  __shared__ const uint32_t* chain[64];
  __shared__ uint32_t msg[64];
  p2_load_full_keys(keys);
  P2Lane L;
  L.init(keys);
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, per = warps * P2_GROUPS_PER_WARP;
  const uint32_t nb = gridDim.x, b = blockIdx.x, first = warp * P2_GROUPS_PER_WARP, group = (uint32_t)L.base / 6;
  auto fold = [&](uint32_t w) {
    uint32_t cnt = 0;
    for (uint32_t t = 0; t < n_inj && cnt < 64; t++)
      if (inj[t].width == w) {
        if (threadIdx.x == 0) chain[cnt] = inj[t].leaves;
        cnt++;
      }
    __syncthreads();
    const uint32_t share = w / nb;
    if (cnt)
      for (uint32_t j0 = first; j0 < share; j0 += per) {
        const uint32_t jl = j0 + group, j = b * share + jl;
        merkle_chain(nodes, (uint64_t)w + j, j, chain, cnt, L, keys, L.lane < 30 && jl < share);
      }
    __syncthreads();
  };
  if (fold_first) fold(top);
  for (uint32_t w = top >> 1; w >= nb; w >>= 1) {
    const uint32_t share = w / nb;
    for (uint32_t i0 = first; i0 < share; i0 += per) {  // a warp without a node skips the level
      const uint32_t il = i0 + group;
      merkle_node(nodes, (uint64_t)w + b * share + il, L, keys, L.lane < 30 && il < share);
    }
    __syncthreads();
    fold(w);
  }
  if (fs.out && warp == 0) {  // the root is nodes[1], written before the last barrier
    const uint32_t total = fs.n_pre + 16;
    for (uint32_t i = L.lane; i < total; i += 32)
      msg[i] = i < fs.n_pre ? fs.pre[i] : (i < fs.n_pre + 8 ? fs.prev[i - fs.n_pre] : nodes[8 + i - fs.n_pre - 8]);
    __syncwarp();
    uint32_t x[4] = {0, 0, 0, 0};
    for (uint32_t b0 = 0; b0 < total; b0 += 16) {
      const uint32_t len = min(16u, total - b0);
      if (L.idx < 4)
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (4 * (uint32_t)L.idx + k < len) x[k] = msg[b0 + 4 * L.idx + k];
      p2c_permute(x, L, keys);
    }
    if (L.lane < 2)
#pragma unroll
      for (int k = 0; k < 4; k++) fs.out[4 * L.lane + k] = x[k];
  }
}

// Permutations of states of 24 words: one state per group of six lanes, and
// one per thread for as many states as occupy the GPU so (p2_per_thread).
__global__ void k_p2_permute(uint32_t* states, uint64_t n) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(4)];
  p2_load_full_keys(keys);
  P2Lane L;
  L.init(keys);
  const uint64_t warps = blockDim.x >> 5;
  const uint64_t i = (blockIdx.x * warps + (threadIdx.x >> 5)) * P2_GROUPS_PER_WARP + (uint64_t)L.base / 6;
  const bool active = L.lane < 30 && i < n;
  uint32_t x[4] = {0, 0, 0, 0};
  if (active)
    for (int q = 0; q < 4; q++) x[q] = states[i * 24 + 4 * L.idx + q];
  p2c_permute(x, L, keys);
  if (active)
    for (int q = 0; q < 4; q++) states[i * 24 + 4 * L.idx + q] = x[q];
}
__global__ void __launch_bounds__(P2_MAX_BLOCK, 2) k_p2_permute1(uint32_t* states, uint64_t n) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[24];
#pragma unroll
  for (int q = 0; q < 24; q++) s[q] = states[i * 24 + q];
  p2_permute(s);
#pragma unroll
  for (int q = 0; q < 24; q++) states[i * 24 + q] = s[q];
}

// ---------------------------------------------------------------- expressions
// Register bytecode for the constraint DAG (compiled on the host from the
// program's folded relation): typed ops over a per-thread register file of
// E6 slots held in shared memory.
enum : uint8_t {
  X_LOAD_B = 0,  // r[d] = col lane imm at row (j + shift) mod n (base)
  X_LOAD_E,      // r[d] = 6 lanes starting at lane imm (ext)
  X_COIN,        // r[d] = coins[imm]
  X_CONST,       // r[d] = imm (base, Montgomery)
  X_ADD_BB, X_ADD_EB, X_ADD_EE,
  X_SUB_BB, X_SUB_BE, X_SUB_EB, X_SUB_EE,
  X_MUL_BB, X_MUL_EB, X_MUL_EE,
};
struct XInst { uint8_t op, d, a, b; uint32_t imm; int32_t shift; };
constexpr int X_MAX_REGS = 24;
constexpr int X_MAX_INST = 16384;  // instructions are read from global memory; no fixed array

struct XProgram {
  const XInst* code;
  uint32_t n_inst;
  uint32_t n_regs;
  uint32_t result;      // register holding the value
  uint32_t result_ext;  // 1 when the result is an E6
};

// Evaluates one row.  lane(l, row) returns column lane l at `row`.
template <class LaneFn>
__device__ __forceinline__ E6 x_eval(const XProgram& p, const E6* coins, uint32_t* regs, uint32_t stride, uint32_t j,
                                     uint32_t n, LaneFn lane) {
  // regs: register r word w at regs[(r * 6 + w) * stride]
  auto R = [&](uint32_t r, int w) -> uint32_t& { return regs[(r * 6 + w) * stride]; };
  for (uint32_t pc = 0; pc < p.n_inst; pc++) {
    XInst in = p.code[pc];
    switch (in.op) {
      case X_LOAD_B: {
        uint32_t row = (uint32_t)(((int64_t)j + in.shift) & (int64_t)(n - 1));
        R(in.d, 0) = lane(in.imm, row);
        break;
      }
      case X_LOAD_E: {
        uint32_t row = (uint32_t)(((int64_t)j + in.shift) & (int64_t)(n - 1));
        for (int w = 0; w < 6; w++) R(in.d, w) = lane(in.imm + w, row);
        break;
      }
      case X_COIN:
        for (int w = 0; w < 6; w++) R(in.d, w) = coins[in.imm].c[w];
        break;
      case X_CONST: R(in.d, 0) = in.imm; break;
      case X_ADD_BB: R(in.d, 0) = add(R(in.a, 0), R(in.b, 0)); break;
      case X_ADD_EB: {  // a ext, b base
        uint32_t b0 = R(in.b, 0);
        for (int w = 1; w < 6; w++) R(in.d, w) = R(in.a, w);
        R(in.d, 0) = add(R(in.a, 0), b0);
        break;
      }
      case X_ADD_EE: for (int w = 0; w < 6; w++) R(in.d, w) = add(R(in.a, w), R(in.b, w)); break;
      case X_SUB_BB: R(in.d, 0) = sub(R(in.a, 0), R(in.b, 0)); break;
      case X_SUB_BE: {  // a base, b ext
        uint32_t a0 = R(in.a, 0);
        for (int w = 1; w < 6; w++) R(in.d, w) = neg(R(in.b, w));
        R(in.d, 0) = sub(a0, R(in.b, 0));
        break;
      }
      case X_SUB_EB: {
        uint32_t b0 = R(in.b, 0);
        for (int w = 1; w < 6; w++) R(in.d, w) = R(in.a, w);
        R(in.d, 0) = sub(R(in.a, 0), b0);
        break;
      }
      case X_SUB_EE: for (int w = 0; w < 6; w++) R(in.d, w) = sub(R(in.a, w), R(in.b, w)); break;
      case X_MUL_BB: R(in.d, 0) = mul(R(in.a, 0), R(in.b, 0)); break;
      case X_MUL_EB: {
        uint32_t b0 = R(in.b, 0);
        for (int w = 0; w < 6; w++) R(in.d, w) = mul(R(in.a, w), b0);
        break;
      }
      case X_MUL_EE: {
        E6 x, y;
        for (int w = 0; w < 6; w++) { x.c[w] = R(in.a, w); y.c[w] = R(in.b, w); }
        E6 z = e6_mul(x, y);
        for (int w = 0; w < 6; w++) R(in.d, w) = z.c[w];
        break;
      }
    }
  }
  E6 r;
  if (p.result_ext) { for (int w = 0; w < 6; w++) r.c[w] = R(p.result, w); }
  else r = e6_base(R(p.result, 0));
  return r;
}

// Quotient numerator of one module on coset c = blockIdx.y, row j:
// V(...) / (s_c^n - 1), written as qv[w * 4n + c n + j].  cv: coset values,
// lane l coset c at cv[l * 4n + c n + j].  One job per module (blockIdx.z).
struct QJob { XProgram p; const uint32_t* cv; uint32_t* qv; int logn; uint32_t zinv[4]; };
__global__ void k_quotient_eval(const QJob* jobs, const E6* coins) {
  extern __shared__ uint32_t regs[];
  const QJob& J = jobs[blockIdx.z];
  const uint32_t n = 1u << J.logn;
  const uint32_t c = blockIdx.y;
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint64_t big = (uint64_t)n << RATE_LOG;
  const uint32_t* cv = J.cv;
  auto lane = [&](uint32_t l, uint32_t row) -> uint32_t { return cv[l * big + (uint64_t)c * n + row]; };
  E6 v = x_eval(J.p, coins, regs + threadIdx.x, blockDim.x, j, n, lane);
  v = e6_mul_base(v, J.zinv[c]);
  uint32_t lw = J.p.result_ext ? 6 : 1;
  for (uint32_t w = 0; w < lw; w++) J.qv[w * big + (uint64_t)c * n + j] = v.c[w];
}

// Quotient chunk coefficients from the inverse-transformed coset values.
// r[w][c n + k] holds [Y^k] R_c(Y), R_c(Y) = sum_d s_c^(dn) q_d(s_c Y).
// With t_c = r_c[k] s_c^-k, u_d = g^(dn) q_(d,k) = 1/4 sum_c t_c w_4^(-cd).
// out: chunk d, lane w at out[(d * lanes + w) * n + k].  One job per module.
struct QcJob { const uint32_t* r; uint32_t* out; int logn; uint32_t lanes; const uint32_t* ginv_pow; const uint32_t* tw_4n; uint32_t gn_inv; };
__global__ void k_quotient_chunks(const QcJob* jobs, uint32_t quarter) {
  const QcJob& J = jobs[blockIdx.z];
  const uint32_t n = 1u << J.logn;
  const uint64_t big = (uint64_t)n << RATE_LOG;
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t w = blockIdx.y;
  if (k >= n || w >= J.lanes) return;
  uint32_t t[4];
  const uint32_t gk = J.ginv_pow[k];
  for (int c = 0; c < 4; c++) {
    uint32_t e = (uint32_t)((big - ((uint64_t)c * k) % big) % big);  // s_c^-k = g^-k w_4n^-(c k)
    t[c] = mul(mul(J.r[w * big + (uint64_t)c * n + k], gk), __ldg(J.tw_4n + e));
  }
  const uint32_t w4i = __ldg(J.tw_4n + 3 * n), w4i2 = mul(w4i, w4i), w4i3 = mul(w4i2, w4i);
  uint32_t u[4];
  u[0] = add(add(t[0], t[1]), add(t[2], t[3]));
  u[1] = add(add(t[0], mul(t[1], w4i)), add(mul(t[2], w4i2), mul(t[3], w4i3)));
  u[2] = add(add(t[0], mul(t[1], w4i2)), add(t[2], mul(t[3], w4i2)));
  u[3] = add(add(t[0], mul(t[1], w4i3)), add(mul(t[2], w4i2), mul(t[3], w4i)));
  uint32_t scale = quarter;
  for (int d = 0; d < 4; d++) {
    J.out[((uint64_t)d * J.lanes + w) * n + k] = mul(u[d], scale);
    scale = mul(scale, J.gn_inv);
  }
}

// ---------------------------------------------------------------- grand product
// ratio[j] = num(j) / den(j) on Lagrange rows (internal/poly/iop_utils.go:170-192).
// One job per step (blockIdx.y); lanes[l] is lane l of the step's inputs.
struct GpJob { XProgram pn, pd; const uint32_t* const* lanes; uint32_t* ratio; int logn; };
__global__ void k_gp_ratio(const GpJob* jobs, const E6* coins) {
  extern __shared__ uint32_t regs[];
  const GpJob& J = jobs[blockIdx.y];
  const uint32_t n = 1u << J.logn;
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t* const* lanes = J.lanes;
  auto lane = [&](uint32_t l, uint32_t row) -> uint32_t { return lanes[l][row]; };
  E6 a = x_eval(J.pn, coins, regs + threadIdx.x, blockDim.x, j, n, lane);
  E6 b = x_eval(J.pd, coins, regs + threadIdx.x, blockDim.x, j, n, lane);
  E6 q = e6_mul(a, e6_inv(b));
  for (int w = 0; w < 6; w++) J.ratio[(uint64_t)w * n + j] = q.c[w];
}

constexpr int SCAN_BLOCK = 256, SCAN_PER_THREAD = 8, SCAN_TILE = SCAN_BLOCK * SCAN_PER_THREAD;

__device__ __forceinline__ E6 ld6(const uint32_t* p, uint64_t stride, uint64_t i) {
  E6 r;
  for (int w = 0; w < 6; w++) r.c[w] = p[w * stride + i];
  return r;
}
__device__ __forceinline__ void st6(uint32_t* p, uint64_t stride, uint64_t i, const E6& v) {
  for (int w = 0; w < 6; w++) p[w * stride + i] = v.c[w];
}

// Product scans over E6 vectors stored as 6 lanes of n words: per-tile
// inclusive scan in place, tile totals, their exclusive prefix, and the
// shifted result out[0] = 1, out[i] = prod_{k<i} x[k].  One job per vector.
struct ScanJob {
  uint32_t* x;
  uint64_t n;
  uint32_t* totals;
  uint32_t* pre;
  uint32_t* out;
  uint32_t nt;
  uint32_t inclusive = 0;  // running ratio: out[i] = prod_{k<=i} x[k] ...
  uint32_t* end = nullptr; // ... and its last value written here (6 words)
};

template <bool SUM = false>
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_tiles(const ScanJob* jobs) {
  __shared__ E6 sh[SCAN_BLOCK / 32];
  const ScanJob& J = jobs[blockIdx.y];
  if (blockIdx.x >= J.nt) return;
  const uint64_t n = J.n;
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_PER_THREAD;
  E6 acc = scan_id<SUM>();
  E6 v[SCAN_PER_THREAD];
#pragma unroll
  for (int i = 0; i < SCAN_PER_THREAD; i++) {
    if (base + i < n) acc = scan_op<SUM>(acc, ld6(J.x, n, base + i));
    v[i] = acc;
  }
  E6 total;
  const E6 pre = block_scan<SUM, SCAN_BLOCK>(acc, sh, total);
#pragma unroll
  for (int i = 0; i < SCAN_PER_THREAD; i++)
    if (base + i < n) st6(J.x, n, base + i, scan_op<SUM>(pre, v[i]));
  if (threadIdx.x < 6) J.totals[threadIdx.x * J.nt + blockIdx.x] = total.c[threadIdx.x];
}

// Exclusive prefix (products or sums) of the tile totals, one block per job
// (nt is n / 2048: a thread alone took 34 us for the 128 tiles of 2^18 rows).
constexpr int PREFIX_BLOCK = 64;
template <bool SUM = false>
__global__ void __launch_bounds__(PREFIX_BLOCK) k_tile_prefix(const ScanJob* jobs) {
  __shared__ E6 sh[PREFIX_BLOCK / 32];
  const ScanJob& J = jobs[blockIdx.x];
  const uint32_t per = (J.nt + PREFIX_BLOCK - 1) / PREFIX_BLOCK, first = threadIdx.x * per;
  E6 acc = scan_id<SUM>();
  for (uint32_t t = first; t < first + per && t < J.nt; t++) acc = scan_op<SUM>(acc, ld6(J.totals, J.nt, t));
  E6 total;
  acc = block_scan<SUM, PREFIX_BLOCK>(acc, sh, total);
  for (uint32_t t = first; t < first + per && t < J.nt; t++) {
#pragma unroll
    for (int w = 0; w < 6; w++) J.pre[t * 6 + w] = acc.c[w];
    acc = scan_op<SUM>(acc, ld6(J.totals, J.nt, t));
  }
}

__global__ void k_gp_finish(const ScanJob* jobs) {
  const ScanJob& J = jobs[blockIdx.y];
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= J.n) return;
  E6 v;
  if (!J.inclusive && i == 0) v = e6_one();
  else {
    uint64_t k = J.inclusive ? i : i - 1, tile = k / SCAN_TILE;
    E6 pre;
    for (int w = 0; w < 6; w++) pre.c[w] = J.pre[tile * 6 + w];
    v = e6_mul(pre, ld6(J.x, J.n, k));
  }
  st6(J.out, J.n, i, v);
  if (J.end && i == J.n - 1)
    for (int w = 0; w < 6; w++) J.end[w] = v.c[w];
}

// ---------------------------------------------------------------- lookups
// Cyclic logup fractions (internal/poly/iop_utils.go:110-131): per row,
// frac = sum_k M_k / E_k over the step's terms.  One job per step.
constexpr int LOGUP_MAX_TERMS = 4;
struct LogupJob {
  XProgram e[LOGUP_MAX_TERMS], m[LOGUP_MAX_TERMS];
  uint32_t n_terms;
  const uint32_t* const* lanes;
  uint32_t* frac;
  int logn;
};
__global__ void k_logup_frac(const LogupJob* jobs, const E6* coins) {
  extern __shared__ uint32_t regs[];
  const LogupJob& J = jobs[blockIdx.y];
  const uint32_t n = 1u << J.logn;
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t* const* lanes = J.lanes;
  auto lane = [&](uint32_t l, uint32_t row) -> uint32_t { return lanes[l][row]; };
  E6 v = e6_zero();
  for (uint32_t k = 0; k < J.n_terms; k++) {
    E6 e = x_eval(J.e[k], coins, regs + threadIdx.x, blockDim.x, j, n, lane);
    E6 m = x_eval(J.m[k], coins, regs + threadIdx.x, blockDim.x, j, n, lane);
    v = e6_add(v, e6_mul(m, e6_inv(e)));
  }
  for (int w = 0; w < 6; w++) J.frac[(uint64_t)w * n + j] = v.c[w];
}

// L_i = S_i - (i + 1) T / n with S the inclusive running sums (tile scans in
// x plus the tile prefixes) and T = S_{n-1}; thread 0 writes T to `total`
// (board/logup.go:150-170).
struct LogupFinish { uint32_t* total; uint32_t n_inv; };
__global__ void k_logup_finish(const ScanJob* jobs, const LogupFinish* fin) {
  const ScanJob& J = jobs[blockIdx.y];
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= J.n) return;
  auto prefix = [&](uint64_t k) {
    E6 pre;
    for (int w = 0; w < 6; w++) pre.c[w] = J.pre[(k / SCAN_TILE) * 6 + w];
    return e6_add(pre, ld6(J.x, J.n, k));
  };
  const E6 T = prefix(J.n - 1);
  const E6 avg = e6_mul_base(T, fin[blockIdx.y].n_inv);
  const E6 L = e6_sub(prefix(i), e6_mul_base(avg, to_mont((uint32_t)(i + 1))));
  st6(J.out, J.n, i, L);
  if (i == 0)
    for (int w = 0; w < 6; w++) fin[blockIdx.y].total[w] = T.c[w];
}

// Lookup multiplicities of width-1 tables (internal/poly/lookup_multiplicity.go:37-100)
// with an open-addressing table per step: target values are inserted with
// the smallest combined row index (T_0 rows, then T_1 rows, ...) holding them,
// sources add one to the count of their value's first row, and the counts
// become the multiplicity columns.  A source value absent from every target
// sets `missing`.  All probe loops stop after `cap` slots.
constexpr uint32_t MULT_EMPTY = 0xffffffffu;
struct MultTab { uint32_t* keys; uint32_t* first; uint32_t* count; uint32_t cap; };
struct MultVec { const uint32_t* vals; uint32_t n, comb_off, tab; uint32_t* out; };
__device__ __forceinline__ uint32_t mult_hash(uint32_t v, uint32_t mask) {
  v ^= v >> 16;
  v *= 0x7feb352du;
  v ^= v >> 15;
  v *= 0x846ca68bu;
  v ^= v >> 16;
  return v & mask;
}
__global__ void k_mult_insert(const MultVec* tv, const MultTab* tabs) {
  const MultVec V = tv[blockIdx.y];
  const MultTab T = tabs[V.tab];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  const uint32_t key = V.vals[i], mask = T.cap - 1;
  uint32_t h = mult_hash(key, mask);
  for (uint32_t probe = 0; probe < T.cap; probe++, h = (h + 1) & mask) {
    const uint32_t prev = atomicCAS(T.keys + h, MULT_EMPTY, key);
    if (prev == MULT_EMPTY || prev == key) {
      atomicMin(T.first + h, V.comb_off + i);
      return;
    }
  }
}
__global__ void k_mult_count(const MultVec* sv, const MultTab* tabs, uint32_t* missing) {
  const MultVec V = sv[blockIdx.y];
  const MultTab T = tabs[V.tab];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  const uint32_t key = V.vals[i], mask = T.cap - 1;
  uint32_t h = mult_hash(key, mask);
  for (uint32_t probe = 0; probe < T.cap; probe++, h = (h + 1) & mask) {
    const uint32_t k = T.keys[h];
    if (k == key) {
      atomicAdd(T.count + T.first[h], 1u);
      return;
    }
    if (k == MULT_EMPTY) break;
  }
  atomicOr(missing, 1u);
}
__global__ void k_mult_write(const MultVec* tv, const MultTab* tabs) {
  const MultVec V = tv[blockIdx.y];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  V.out[i] = to_mont(tabs[V.tab].count[V.comb_off + i]);
}
// Tuple lookups with selectors (internal/poly/lookup_multiplicity.go:37-100).
// A step's hash table keys tuples by a representative target row whose
// tuple sits in `keys` (w words per combined target row); per slot, the
// first selected target row holding the tuple and the selected source weight
// (sum of canonical selector values, 64-bit).  Probes are bounded by the
// table size, which is at least twice the target rows.
constexpr uint32_t TUPLE_MAX_W = 8;
struct TupleVec { const uint32_t* comp[TUPLE_MAX_W]; const uint32_t* sel; uint32_t n, comb_off, tab; uint32_t* out; };
struct TupleTab { uint32_t* rep; uint32_t* first; unsigned long long* weight; uint32_t* keys; uint32_t cap, w; };
__device__ __forceinline__ uint32_t tuple_hash(const TupleVec& V, uint32_t i, uint32_t w, uint32_t mask) {
  uint32_t h = 0x9e3779b9u;
  for (uint32_t k = 0; k < w; k++) h = mult_hash(h ^ V.comp[k][i], 0xffffffffu) + k;
  return mult_hash(h, mask);
}
__device__ __forceinline__ bool tuple_eq(const TupleVec& V, uint32_t i, const uint32_t* key, uint32_t w) {
  for (uint32_t k = 0; k < w; k++)
    if (V.comp[k][i] != key[k]) return false;
  return true;
}
__global__ void k_tuple_keys(const TupleVec* tv, const TupleTab* tabs) {
  const TupleVec V = tv[blockIdx.y];
  const TupleTab T = tabs[V.tab];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  for (uint32_t k = 0; k < T.w; k++) T.keys[(uint64_t)(V.comb_off + i) * T.w + k] = V.comp[k][i];
}
__global__ void k_tuple_insert(const TupleVec* tv, const TupleTab* tabs, uint32_t* fail) {
  const TupleVec V = tv[blockIdx.y];
  const TupleTab T = tabs[V.tab];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n || (V.sel && V.sel[i] == 0)) return;
  const uint32_t g = V.comb_off + i, mask = T.cap - 1;
  uint32_t h = tuple_hash(V, i, T.w, mask);
  for (uint32_t probe = 0; probe < T.cap; probe++, h = (h + 1) & mask) {
    const uint32_t prev = atomicCAS(T.rep + h, MULT_EMPTY, g);
    if (prev == MULT_EMPTY || tuple_eq(V, i, T.keys + (uint64_t)prev * T.w, T.w)) {
      atomicMin(T.first + h, g);
      return;
    }
  }
  atomicOr(fail, 2u);
}
__global__ void k_tuple_count(const TupleVec* sv, const TupleTab* tabs, uint32_t* missing) {
  const TupleVec V = sv[blockIdx.y];
  const TupleTab T = tabs[V.tab];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  const uint32_t sel = V.sel ? V.sel[i] : MONT_ONE;
  if (sel == 0) return;
  const uint32_t mask = T.cap - 1;
  uint32_t h = tuple_hash(V, i, T.w, mask);
  for (uint32_t probe = 0; probe < T.cap; probe++, h = (h + 1) & mask) {
    const uint32_t r = T.rep[h];
    if (r == MULT_EMPTY) break;
    if (tuple_eq(V, i, T.keys + (uint64_t)r * T.w, T.w)) {
      atomicAdd(T.weight + h, (unsigned long long)from_mont(sel));
      return;
    }
  }
  atomicOr(missing, 1u);
}
__global__ void k_tuple_write(const TupleVec* tv, const TupleTab* tabs) {
  const TupleVec V = tv[blockIdx.y];
  const TupleTab T = tabs[V.tab];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  uint32_t m = 0;
  const uint32_t sel = V.sel ? V.sel[i] : MONT_ONE;
  if (sel != 0) {
    const uint32_t g = V.comb_off + i, mask = T.cap - 1;
    uint32_t h = tuple_hash(V, i, T.w, mask);
    for (uint32_t probe = 0; probe < T.cap; probe++, h = (h + 1) & mask) {
      const uint32_t r = T.rep[h];
      if (r == MULT_EMPTY) break;
      if (tuple_eq(V, i, T.keys + (uint64_t)r * T.w, T.w)) {
        if (T.first[h] == g) m = mul(to_mont((uint32_t)(T.weight[h] % P)), V.sel ? inv(sel) : MONT_ONE);
        break;
      }
    }
  }
  V.out[i] = m;
}

// Values of a base-field expression on every row (for lookup tables that are
// not plain columns).
struct EvalJob { XProgram p; const uint32_t* const* lanes; uint32_t* out; int logn; };
__global__ void k_eval_base(const EvalJob* jobs, const E6* coins) {
  extern __shared__ uint32_t regs[];
  const EvalJob& J = jobs[blockIdx.y];
  const uint32_t n = 1u << J.logn;
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t* const* lanes = J.lanes;
  auto lane = [&](uint32_t l, uint32_t row) -> uint32_t { return lanes[l][row]; };
  J.out[j] = x_eval(J.p, coins, regs + threadIdx.x, blockDim.x, j, n, lane).c[0];
}

// ---------------------------------------------------------------- claimed values
// P(z) of base lanes from their coefficients, z = zeta w_n^s.  A thread takes
// EVAL_RUN consecutive coefficients: sum_j c_(16 i + j) z^j with the 16 low
// powers shared by the whole launch, then one E6 product by z^(16 i).
//
// What bounds it: the integer-multiply pipe, 6 wide products a coefficient
// summed four at a time before their reduction (mont_reduce4), plus a
// sixteenth of an E6 product; the coefficients are read once (4 B against 28 B
// a coefficient with a table of every power), and a lane is cut into chunks
// so that a long one does not end up in one block.  B200, ten modules of
// 2^10 .. 2^18 rows, 767 evaluations: 0.13 ms of powers and sums together,
// where a table of every power (0.69 ms) and a block per evaluation (1.55 ms)
// were before; 40 modules of 2^14 rows, 2000 evaluations: 0.08 ms (0.20 ms).
constexpr int EVAL_RUN = 16, EVAL_BLOCK = 256, EVAL_TURNS = 2;
constexpr uint32_t EVAL_CHUNK = EVAL_RUN * EVAL_BLOCK * EVAL_TURNS;  // coefficients per block

// One evaluation point of a size: lo[6 j + w] = z^j (j < 16), hi[w m + i] =
// z^(16 i) (i < m = max(1, n/16)).
struct EvalPoint { uint32_t ws; uint32_t m; uint32_t* lo; uint32_t* hi; };
constexpr int EVAL_POW_BLOCK = 128, EVAL_POW_TURNS = 8;
__global__ void __launch_bounds__(EVAL_POW_BLOCK) k_eval_powers(const EvalPoint* points, const uint32_t* zeta_w) {
  const EvalPoint pt = points[blockIdx.x];
  const uint32_t first = blockIdx.y * EVAL_POW_BLOCK * EVAL_POW_TURNS;
  if (first >= pt.m) return;
  E6 z;
#pragma unroll
  for (int w = 0; w < 6; w++) z.c[w] = zeta_w[w];
  z = e6_mul_base(z, pt.ws);
  if (blockIdx.y == 0 && threadIdx.x < EVAL_RUN) {
    const E6 v = e6_pow(z, threadIdx.x);
#pragma unroll
    for (int w = 0; w < 6; w++) pt.lo[6 * threadIdx.x + w] = v.c[w];
  }
  static_assert(EVAL_RUN == 16, "four squarings");
#pragma unroll 1
  for (int k = 0; k < 4; k++) z = e6_sqr(z);
  E6 v = e6_pow(z, first + threadIdx.x);
  if (pt.m > first + EVAL_POW_BLOCK) {
#pragma unroll 1
    for (int k = EVAL_POW_BLOCK; k > 1; k >>= 1) z = e6_sqr(z);
  }
  for (int t = 0; t < EVAL_POW_TURNS; t++) {
    const uint32_t i = first + t * EVAL_POW_BLOCK + threadIdx.x;
    if (i >= pt.m) return;
    st6(pt.hi, pt.m, i, v);
    v = e6_mul(v, z);
  }
}

// Block (job, chunk): the sum over the chunk's coefficients, to out (one chunk)
// or to part, 6 words each.
struct EvalLaneJob { const uint32_t* coef; uint32_t n, point, part; };  // part: index of its first chunk's sum
__global__ void __launch_bounds__(EVAL_BLOCK, 2) k_eval_lanes(const EvalLaneJob* jobs, const EvalPoint* points,
                                                              uint32_t* part, uint32_t* out) {
  const EvalLaneJob jb = jobs[blockIdx.x];
  const uint32_t first = blockIdx.y * EVAL_CHUNK;
  if (first >= jb.n) return;
  const EvalPoint pt = points[jb.point];
  __shared__ __align__(16) uint32_t lo[6 * EVAL_RUN];
  __shared__ E6 warp_sum[EVAL_BLOCK / 32];
  if (threadIdx.x < 6 * EVAL_RUN) lo[threadIdx.x] = pt.lo[threadIdx.x];
  __syncthreads();
  E6 sum = e6_zero();
  const bool aligned = ((uintptr_t)jb.coef & 15) == 0;
#pragma unroll 1
  for (int turn = 0; turn < EVAL_TURNS; turn++) {
    const uint32_t i = first / EVAL_RUN + turn * EVAL_BLOCK + threadIdx.x;
    if (i >= pt.m) break;
    const uint32_t k0 = i * EVAL_RUN;
    uint32_t c[EVAL_RUN];
    if (aligned && k0 + EVAL_RUN <= jb.n) {
#pragma unroll
      for (int q = 0; q < EVAL_RUN / 4; q++) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(jb.coef + k0) + q);
        c[4 * q] = v.x;
        c[4 * q + 1] = v.y;
        c[4 * q + 2] = v.z;
        c[4 * q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < EVAL_RUN; q++) c[q] = k0 + q < jb.n ? __ldg(jb.coef + k0 + q) : 0u;
    }
    E6 v = e6_zero();
#pragma unroll
    for (int q = 0; q < EVAL_RUN; q += 4) {
      const uint4* l4 = reinterpret_cast<const uint4*>(lo + 6 * q);  // z^q .. z^(q+3), 24 words
      uint32_t l[24];
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const uint4 x = l4[k];
        l[4 * k] = x.x;
        l[4 * k + 1] = x.y;
        l[4 * k + 2] = x.z;
        l[4 * k + 3] = x.w;
      }
#pragma unroll
      for (int w = 0; w < 6; w++) {
        uint64_t t = (uint64_t)c[q] * l[w];
        t += (uint64_t)c[q + 1] * l[6 + w];
        t += (uint64_t)c[q + 2] * l[12 + w];
        t += (uint64_t)c[q + 3] * l[18 + w];
        v.c[w] = add(v.c[w], mont_reduce4(t));
      }
    }
    sum = e6_add(sum, pt.m > 1 ? e6_mul(v, ld6(pt.hi, pt.m, i)) : v);
  }
  // the block's sum
#pragma unroll
  for (int w = 0; w < 6; w++)
    for (int off = 16; off; off >>= 1) sum.c[w] = add(sum.c[w], __shfl_xor_sync(0xffffffffu, sum.c[w], off));
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 6) {
    uint32_t s = 0;
    for (int k = 0; k < EVAL_BLOCK / 32; k++) s = add(s, warp_sum[k].c[threadIdx.x]);
    uint32_t* dst = jb.n <= EVAL_CHUNK ? out + 6 * (uint64_t)blockIdx.x : part + 6 * ((uint64_t)jb.part + blockIdx.y);
    dst[threadIdx.x] = s;
  }
}
// The chunks' sums of the jobs longer than one chunk: a warp per job.
__global__ void __launch_bounds__(32) k_eval_sum(const EvalLaneJob* jobs, const uint32_t* part, uint32_t* out) {
  const EvalLaneJob jb = jobs[blockIdx.x];
  if (jb.n <= EVAL_CHUNK) return;
  const uint32_t chunks = (jb.n + EVAL_CHUNK - 1) / EVAL_CHUNK;
  E6 s = e6_zero();
  for (uint32_t k = threadIdx.x; k < chunks; k += 32)
#pragma unroll
    for (int w = 0; w < 6; w++) s.c[w] = add(s.c[w], part[6 * ((uint64_t)jb.part + k) + w]);
#pragma unroll
  for (int w = 0; w < 6; w++)
    for (int off = 16; off; off >>= 1) s.c[w] = add(s.c[w], __shfl_xor_sync(0xffffffffu, s.c[w], off));
  if (threadIdx.x == 0)
#pragma unroll
    for (int w = 0; w < 6; w++) out[6 * (uint64_t)blockIdx.x + w] = s.c[w];
}

// ---------------------------------------------------------------- DEEP
// DQ(x) = sum_s (A_s - sum_{b in s} alpha^i_b P_b(x)) / (z_s - x) on the LDE
// rows r of one class, x = w_4n^bitrev(r) (internal/fri/deep.go:205-266,
// evaluated on the 4n LDE rows instead of the n trace rows and re-encoded:
// DQ has degree < n, so both give the same codeword).
constexpr int DEEP_MAX_POINTS = 4;
// Every polynomial enters as base lanes with an E6 coefficient each (an
// extension polynomial as its six lanes, alpha^i times the basis elements), so
// a row's sum is one dot product over the lanes of the class.  Lanes are
// sorted by the set of points they are opened at (`mask`) and padded to whole
// quads of one mask with zero coefficients: four products are summed before
// each reduction (mont_reduce4).
struct DeepLane { const uint32_t* p; uint32_t c[6]; uint32_t mask, pad; };
struct DeepJob {
  const DeepLane* lanes;
  uint32_t n_lanes;     // a multiple of four
  uint32_t n_points;
  E6 z[DEEP_MAX_POINTS];
  const uint32_t* a;    // the points' weighted values, six words each (device)
  int logn4;            // log2 of the LDE size
  uint32_t vec;         // lanes aligned to the rows a thread takes
  const uint32_t* tw;   // w_4n^j table
  uint32_t* out;        // 6 lanes, lane stride 4n; or rows of six words
  const uint32_t* den;  // 1/(z_s - x) from k_deep_den (null: computed here)
};

// The DEEP denominators 1/(z_s - x) of every LDE row r of a class (x =
// w_4n^bitrev(r)), one inversion per row for all its points (Montgomery's
// trick), stored as six lanes per point: den[(6 s + w) 4n + r].  z_s =
// zeta ws[s] with zeta read from its device slot, so the kernel runs as
// soon as zeta is known, beside the claimed values and the host's
// alpha_DEEP transcript.
struct DenJob { uint32_t n_points; uint32_t ws[DEEP_MAX_POINTS]; int logn4; const uint32_t* tw; uint32_t* den; };
__global__ void k_deep_den(const DenJob* jobs, const uint32_t* zeta_w) {
  const DenJob& jb = jobs[blockIdx.y];
  const uint32_t big = 1u << jb.logn4;
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= big) return;
  E6 zeta;
#pragma unroll
  for (int w = 0; w < 6; w++) zeta.c[w] = zeta_w[w];
  const uint32_t x = __ldg(jb.tw + bitrev32(r, jb.logn4));
  const uint32_t np = jb.n_points;
  E6 d[DEEP_MAX_POINTS], pre[DEEP_MAX_POINTS];
  for (uint32_t s = 0; s < np; s++) {
    d[s] = e6_mul_base(zeta, jb.ws[s]);
    d[s].c[0] = sub(d[s].c[0], x);
    pre[s] = s ? e6_mul(pre[s - 1], d[s]) : d[s];
  }
  auto put = [&](uint32_t s, const E6& v) {
#pragma unroll
    for (int w = 0; w < 6; w++) jb.den[(uint64_t)(6 * s + w) * big + r] = v.c[w];
  };
  E6 inv_run = e6_inv(pre[np - 1]);
  for (uint32_t s = np - 1; s > 0; s--) {
    put(s, e6_mul(inv_run, pre[s - 1]));
    inv_run = e6_mul(inv_run, d[s]);
  }
  put(0, inv_run);
}
// ROWS consecutive rows of a lane.
template <int ROWS> __device__ __forceinline__ void ld_rows(const uint32_t* p, bool vec, uint32_t* x) {
  if (vec) {
    if constexpr (ROWS == 4) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
      x[0] = v.x;
      x[1] = v.y;
      x[2] = v.z;
      x[3] = v.w;
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      x[0] = v.x;
      x[1] = v.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < ROWS; i++) x[i] = __ldg(p + i);
  }
}

// 1/(z - x_i) for ROWS values x_i: the parts of e6_inv that hold z's second
// and third coefficient are the same for all of them, and the base-field
// inversions share one (Montgomery's trick; a zero norm, z = x_i, gives 0 as
// inv(0) does).
template <int ROWS> __device__ __forceinline__ void deep_inverses(const E6& z, const uint32_t* x, E6* out) {
  const E2 a1 = g2(z, 1), a2 = g2(z, 2);
  const E2 k1 = e2_mul_xi(e2_mul(a1, a2)), k2 = e2_mul_xi(e2_mul(a2, a2)), k3 = e2_mul(a1, a1);
  // t = a0 (a0^2 - 3 k1) + k4, k4 = xi (a2 k2 + a1 k3)
  const E2 k4 = e2_mul_xi(e2_add(e2_mul(a2, k2), e2_mul(a1, k3)));
  const E2 k13 = {triple(k1.a0), triple(k1.a1)};
  E2 t[ROWS];
  uint32_t norm[ROWS], pre[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; i++) {
    const E2 a0 = {sub(z.c[0], x[i]), z.c[1]};
    t[i] = e2_add(e2_mul(a0, e2_sub(e2_mul(a0, a0), k13)), k4);
    norm[i] = sub(sqr(t[i].a0), triple(sqr(t[i].a1)));
    pre[i] = norm[i] ? norm[i] : MONT_ONE;
    if (i) pre[i] = mul(pre[i], pre[i - 1]);
  }
  uint32_t run = inv(pre[ROWS - 1]);
#pragma unroll
  for (int i = ROWS - 1; i >= 0; i--) {
    uint32_t ni = i ? mul(run, pre[i - 1]) : run;
    run = mul(run, norm[i] ? norm[i] : MONT_ONE);
    if (!norm[i]) ni = 0;
    const E2 ti = {mul(t[i].a0, ni), mul(neg(t[i].a1), ni)};
    const E2 a0 = {sub(z.c[0], x[i]), z.c[1]};
    s2(out[i], 0, e2_mul(e2_sub(e2_mul(a0, a0), k1), ti));
    s2(out[i], 1, e2_mul(e2_sub(k2, e2_mul(a0, a1)), ti));
    s2(out[i], 2, e2_mul(e2_sub(k3, e2_mul(a0, a2)), ti));
  }
}

// DEEP quotients, ROWS consecutive rows per thread; the lanes' pointers and
// coefficients are staged in shared memory.  ROWMAJOR: rows of six words out,
// one point, the denominators computed here.  NP: points held in registers
// (at least the job's).
// What bounds it: the integer-multiply pipe (6 wide products per lane and row;
// 77% of its peak, DRAM 27%).  48 lanes of 2^20 rows on B200: 128 us a call (349 us lane by lane, with the
// points' sums in local memory and a transposing pass after it).
constexpr int DEEP_BLOCK = 128, DEEP_STAGE = 64;
template <int NP, int ROWS, bool ROWMAJOR>
__global__ void __launch_bounds__(DEEP_BLOCK) k_deep(const DeepJob* jobs) {
  __shared__ __align__(16) DeepLane sh[DEEP_STAGE];
  const DeepJob& jb = jobs[blockIdx.y];
  const uint32_t big = 1u << jb.logn4;
  if (blockIdx.x * (uint32_t)(DEEP_BLOCK * ROWS) >= big) return;
  const uint32_t r = (blockIdx.x * DEEP_BLOCK + threadIdx.x) * ROWS;
  const bool in = r < big, vec = jb.vec != 0;
  E6 acc[NP][ROWS];
#pragma unroll
  for (int s = 0; s < NP; s++)
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
      acc[s][i] = e6_zero();
      if ((uint32_t)s < jb.n_points)
#pragma unroll
        for (int w = 0; w < 6; w++) acc[s][i].c[w] = jb.a[6 * s + w];
    }
  E6 sum[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; i++) sum[i] = e6_zero();
  uint32_t mask = 0;
  auto flush = [&]() {
#pragma unroll
    for (int s = 0; s < NP; s++)
      if (mask >> s & 1)
#pragma unroll
        for (int i = 0; i < ROWS; i++) acc[s][i] = e6_sub(acc[s][i], sum[i]);
#pragma unroll
    for (int i = 0; i < ROWS; i++) sum[i] = e6_zero();
  };
  for (uint32_t l0 = 0; l0 < jb.n_lanes; l0 += DEEP_STAGE) {
    const uint32_t cnt = min((uint32_t)DEEP_STAGE, jb.n_lanes - l0);
    constexpr uint32_t W = sizeof(DeepLane) / 4;
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cnt * W; k += DEEP_BLOCK)
      reinterpret_cast<uint32_t*>(sh)[k] = reinterpret_cast<const uint32_t*>(jb.lanes + l0)[k];
    __syncthreads();
    if (!in) continue;
    uint32_t next[4][ROWS];  // the next quad's rows, loaded beside this one's products
#pragma unroll
    for (int k = 0; k < 4; k++) ld_rows<ROWS>(sh[k].p + r, vec, next[k]);
#pragma unroll 1
    for (uint32_t q = 0; q < cnt; q += 4) {
      if (sh[q].mask != mask) {
        flush();
        mask = sh[q].mask;
      }
      uint32_t x[4][ROWS];
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int i = 0; i < ROWS; i++) x[k][i] = next[k][i];
      if (q + 4 < cnt)
#pragma unroll
        for (int k = 0; k < 4; k++) ld_rows<ROWS>(sh[q + 4 + k].p + r, vec, next[k]);
#pragma unroll
      for (int w = 0; w < 6; w += 2) {
        uint2 c[4];
#pragma unroll
        for (int k = 0; k < 4; k++) c[k] = *reinterpret_cast<const uint2*>(sh[q + k].c + w);
#pragma unroll
        for (int i = 0; i < ROWS; i++) {
          uint64_t t = (uint64_t)x[0][i] * c[0].x, u = (uint64_t)x[0][i] * c[0].y;
#pragma unroll
          for (int k = 1; k < 4; k++) {
            t += (uint64_t)x[k][i] * c[k].x;
            u += (uint64_t)x[k][i] * c[k].y;
          }
          sum[i].c[w] = add(sum[i].c[w], mont_reduce4(t));
          sum[i].c[w + 1] = add(sum[i].c[w + 1], mont_reduce4(u));
        }
      }
    }
  }
  if (!in) return;
  flush();
  const uint32_t np = jb.n_points;
  E6 dq[ROWS];
  // x of row r + i: w_4n^bitrev(r + i) = w_4n^bitrev(r) w_ROWS^bitrev(i)
  uint32_t x[ROWS];
  if (ROWMAJOR || !jb.den) {
    x[0] = __ldg(jb.tw + bitrev32(r, jb.logn4));
#pragma unroll
    for (int i = 1; i < ROWS; i++) x[i] = __ldg(jb.tw + bitrev32(r + i, jb.logn4));
  }
  if constexpr (ROWMAJOR) {
    E6 di[ROWS];
    deep_inverses<ROWS>(jb.z[0], x, di);
#pragma unroll
    for (int i = 0; i < ROWS; i++) dq[i] = e6_mul(acc[0][i], di[i]);
    uint32_t* o = jb.out + 6 * (uint64_t)r;
    if (vec && ROWS == 4 && ((uintptr_t)jb.out & 15) == 0) {
      const uint32_t* v = reinterpret_cast<const uint32_t*>(dq);
#pragma unroll
      for (int k = 0; k < 6 * ROWS / 4; k++)
        reinterpret_cast<uint4*>(o)[k] = make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < ROWS; i++)
#pragma unroll
        for (int w = 0; w < 6; w++) o[6 * i + w] = dq[i].c[w];
    }
  } else {
    bool pole[ROWS];  // a row at one of the points: 0, as an inversion shared by the points gives
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
      dq[i] = e6_zero();
      pole[i] = false;
    }
#pragma unroll
    for (int s = 0; s < NP; s++) {
      if (s >= np) break;
      E6 di[ROWS];
      if (jb.den) {
#pragma unroll
        for (int w = 0; w < 6; w++) {
          uint32_t d[ROWS];
          ld_rows<ROWS>(jb.den + (uint64_t)(6 * s + w) * big + r, vec, d);
#pragma unroll
          for (int i = 0; i < ROWS; i++) di[i].c[w] = d[i];
        }
      } else {
        deep_inverses<ROWS>(jb.z[s], x, di);
      }
#pragma unroll
      for (int i = 0; i < ROWS; i++) {
        dq[i] = e6_add(dq[i], e6_mul(acc[s][i], di[i]));
        pole[i] |= e6_is_zero(di[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < ROWS; i++)
      if (pole[i]) dq[i] = e6_zero();
#pragma unroll
    for (int w = 0; w < 6; w++) {
      uint32_t* o = jb.out + (uint64_t)w * big + r;
      if (vec && ROWS == 2) *reinterpret_cast<uint2*>(o) = make_uint2(dq[0].c[w], dq[ROWS - 1].c[w]);
      else
#pragma unroll
        for (int i = 0; i < ROWS; i++) o[i] = dq[i].c[w];
    }
  }
}

// The coefficients alpha^i of n columns in the lanes' table and
// a = sum_i alpha^i values[i], one block.
__global__ void __launch_bounds__(256) k_deep_coefs(E6 alpha, const uint32_t* values, uint32_t n, DeepLane* lanes,
                                                    uint32_t* a) {
  __shared__ E6 sh[8];
  E6 step = alpha, v = e6_pow(alpha, threadIdx.x), sum = e6_zero();
#pragma unroll 1
  for (int k = 0; k < 8; k++) step = e6_sqr(step);  // alpha^256
  for (uint32_t i = threadIdx.x; i < n; i += 256) {
#pragma unroll
    for (int w = 0; w < 6; w++) lanes[i].c[w] = v.c[w];
    sum = e6_add(sum, e6_mul(v, ld6(values + 6 * (uint64_t)i, 1, 0)));
    v = e6_mul(v, step);
  }
  E6 total;
  block_scan<true, 256>(sum, sh, total);
  if (threadIdx.x < 6) a[threadIdx.x] = total.c[threadIdx.x];
}

// The weights of a class (a block each), once alpha_DEEP is known: lane l of
// polynomial i gets alpha^i times the basis element of its place `w` (1, u, v,
// u v, v^2, u v^2; padding lanes nothing), and point k gets
// a_k = sum_i alpha^i value(i, k) over the claimed values where the evaluation
// left them (an extension polynomial's as its six lanes).
//
// A chain of E6 products is all that it costs, so the first powers of alpha
// go into a table by doubling (one product a round), and a point's terms are
// summed by a warp.
constexpr uint32_t DEEP_NO_POLY = 0xffffffffu;
struct DeepPlace { uint32_t poly, w; };
struct DeepTerm { uint32_t eval, poly, ext, point; };
struct DeepWeights {
  DeepLane* lanes;
  const DeepPlace* places;
  const DeepTerm* terms;
  uint32_t n_lanes, n_terms, n_points, n_polys;
  uint32_t* a;
};
__device__ __forceinline__ E6 e6_mul_basis(E6 x, uint32_t w) {
  if (w & 1) x = e6_mul_u(x);
  for (uint32_t k = 0; k < w / 2; k++) x = e6_mul_v(x);
  return x;
}
__global__ void __launch_bounds__(128) k_deep_weights(const DeepWeights* classes, E6 alpha, const uint32_t* evals) {
  __shared__ E6 pw[129];
  const DeepWeights cl = classes[blockIdx.x];
  const uint32_t tid = threadIdx.x;
  if (tid < 2) pw[tid] = tid ? alpha : e6_one();
  __syncthreads();
  for (uint32_t d = 1; d < 128 && d < cl.n_polys; d *= 2) {  // alpha^0 .. alpha^d are there
    if (tid < d) pw[d + 1 + tid] = e6_mul(pw[d], pw[1 + tid]);
    __syncthreads();
  }
  auto power = [&](uint32_t i) {
    return i < 128 ? pw[i] : e6_mul(pw[i & 127], e6_pow(pw[128], i >> 7));
  };
  for (uint32_t l = tid; l < cl.n_lanes; l += 128) {
    const DeepPlace pl = cl.places[l];
    const E6 v = pl.poly == DEEP_NO_POLY ? e6_zero() : e6_mul_basis(power(pl.poly), pl.w);
#pragma unroll
    for (int w = 0; w < 6; w++) cl.lanes[l].c[w] = v.c[w];
  }
  for (uint32_t k = tid / 32; k < cl.n_points; k += 4) {
    E6 sum = e6_zero();
    for (uint32_t i = tid % 32; i < cl.n_terms; i += 32) {
      const DeepTerm t = cl.terms[i];
      if (t.point != k) continue;
      E6 v = ld6(evals + 6 * (uint64_t)t.eval, 1, 0);
      if (t.ext)
        for (uint32_t w = 1; w < 6; w++) v = e6_add(v, e6_mul_basis(ld6(evals + 6 * ((uint64_t)t.eval + w), 1, 0), w));
      sum = e6_add(sum, e6_mul(power(t.poly), v));
    }
#pragma unroll
    for (int d = 16; d; d /= 2) {
      E6 o;
#pragma unroll
      for (int w = 0; w < 6; w++) o.c[w] = __shfl_xor_sync(0xffffffffu, sum.c[w], d);
      sum = e6_add(sum, o);
    }
    if (tid % 32 == 0) {
#pragma unroll
      for (int w = 0; w < 6; w++) cl.a[6 * k + w] = sum.c[w];
    }
  }
}

// ---------------------------------------------------------------- FRI
// running += sum_t gamma_t * level_t (6 lanes each, lane stride n), the
// levels entering FRI at this round in level order.
// gamma: device words (the first six words of the challenge's digest).
struct AxpyTerm { const uint32_t* lvl; const uint32_t* gamma; };
__device__ __forceinline__ E6 ld_e6w(const uint32_t* w) {
  E6 r;
#pragma unroll
  for (int k = 0; k < 6; k++) r.c[k] = w[k];
  return r;
}
__global__ void k_axpy_e6(uint32_t* run, uint64_t n, const AxpyTerm* terms, uint32_t n_terms) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  E6 a = ld6(run, n, i);
  for (uint32_t t = 0; t < n_terms; t++) a = e6_add(a, e6_mul(ld6(terms[t].lvl, n, i), ld_e6w(terms[t].gamma)));
  st6(run, n, i, a);
}

// next[i] = (p+q)/2 + alpha (p-q)/(2 x_i), x_i^-1 = w_n^-bitrev(i, n/2)
// (internal/fri/fri.go:1113-1118,1177-1198).  tw: w_n^j table.
// alpha: device words (the first six words of a challenge digest).
__global__ void k_fold(const uint32_t* layer, uint64_t n, const uint32_t* alpha_w, const uint32_t* tw, uint32_t inv2,
                       uint32_t* next) {
  const uint64_t half = n / 2;
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= half) return;
  E6 alpha;
#pragma unroll
  for (int w = 0; w < 6; w++) alpha.c[w] = __ldg(alpha_w + w);
  int lg = 0;
  while ((1ull << lg) < half) lg++;
  uint32_t e = bitrev32((uint32_t)i, lg);
  uint32_t xinv = __ldg(tw + ((n - e) & (n - 1)));
  E6 p = ld6(layer, n, 2 * i), q = ld6(layer, n, 2 * i + 1);
  E6 s = e6_mul_base(e6_add(p, q), inv2);
  E6 d = e6_mul(e6_mul_base(e6_mul_base(e6_sub(p, q), inv2), xinv), alpha);
  st6(next, half, i, e6_add(s, d));
}

// The same fold on rows of six words (ext.E6 arrays, one after another), as
// callers hold them: a thread reads rows 2i and 2i + 1 (48 contiguous bytes)
// and writes row i, so the layer crosses memory once.  x_i^-1 comes from two
// tables that stay in L1 (mul_split, ntt_large.cuh: w_n^-e = w_n^(n - e))
// rather than a scattered read of a table as long as the layer.  VEC: 16- and
// 8-byte accesses (the caller's rows aligned to 16 bytes).
// What bounds it: the multiply pipe, then HBM (an extension product and twelve
// Shoup products for 72 B per output row: 71% and 45% of their peaks).  2^22
// rows on B200: 48 us a call, 0.48 of the
// measured HBM rate (257 us with a copy in, a transpose, the fold, a transpose
// back and a copy out).
constexpr int FOLD_SPLIT = 11;
struct FoldArgs { E6 alpha; const uint2* tw; uint32_t logn; };
template <bool VEC>
__global__ void __launch_bounds__(256) k_fold_rows(const uint32_t* layer, FoldArgs a, uint32_t* next) {
  const uint32_t half = 1u << (a.logn - 1);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= half) return;
  E6 p, q;
  const uint32_t* src = layer + 12 * (uint64_t)i;
  if constexpr (VEC) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(src)), y = __ldg(reinterpret_cast<const uint4*>(src) + 1),
                z = __ldg(reinterpret_cast<const uint4*>(src) + 2);
    p = E6{{x.x, x.y, x.z, x.w, y.x, y.y}};
    q = E6{{y.z, y.w, z.x, z.y, z.z, z.w}};
  } else {
#pragma unroll
    for (int w = 0; w < 6; w++) {
      p.c[w] = src[w];
      q.c[w] = src[6 + w];
    }
  }
  // (p - q)/2 x^-1, then (p + q)/2 + alpha of it
  const uint32_t e = ((1u << a.logn) - bitrev32(i, (int)a.logn - 1)) & ((1u << a.logn) - 1);
  const uint2 lo = __ldg(a.tw + (e & ((1u << FOLD_SPLIT) - 1))), hi = __ldg(a.tw + (1u << FOLD_SPLIT) + (e >> FOLD_SPLIT));
  E6 s, d;
#pragma unroll
  for (int w = 0; w < 6; w++) {
    s.c[w] = mul_pow2_inv<1, false>(p.c[w] + q.c[w]);
    d.c[w] = mulc(mulc_lazy(mul_pow2_inv<1, false>(sub_lazy(p.c[w], q.c[w])), lo.x, lo.y), hi.x, hi.y);
  }
  const E6 v = e6_add(s, e6_mul(d, a.alpha));
  uint32_t* dst = next + 6 * (uint64_t)i;
  if constexpr (VEC) {
    uint2* o = reinterpret_cast<uint2*>(dst);
    o[0] = make_uint2(v.c[0], v.c[1]);
    o[1] = make_uint2(v.c[2], v.c[3]);
    o[2] = make_uint2(v.c[4], v.c[5]);
  } else {
#pragma unroll
    for (int w = 0; w < 6; w++) dst[w] = v.c[w];
  }
}

// The last FRI rounds in one block: for each round j, the fold of layer j
// with challenge j (as k_fold), the levels that enter at j + 1 (as
// k_axpy_e6), then, unless j is the last round, layer j + 1's commitment —
// pair leaves (one permutation each, as k_hash_leaves), the tree level by
// level — and challenge j + 1 from its root (as k_fs_challenge).  Every value
// is written where the per-round launches write it.  Six lanes per
// permutation, five permutations per warp; a warp without a permutation
// leaves the schedulers to the others.
// What bounds it: the latency of 3 + log2(leaves) dependent permutations a
// round (2.7 us each); three launches a round add their starts to that.
constexpr int FRI_TAIL_BLOCK = 512;
struct FriRound {
  const uint32_t* cur;     // layer j: 6 lanes of n words (bit-reversed rows)
  uint32_t* next;          // layer j + 1: 6 lanes of n / 2 words
  const uint32_t* tw;      // w_n^k, k < n
  uint32_t* nodes;         // layer j + 1's tree (2 leaves digests, 1-indexed); null after the last fold
  uint64_t n;              // rows of layer j
  uint32_t log_leaves;     // of that tree
  uint32_t pre_off, pre_len;      // challenge j + 1's name elements in `pre`
  uint32_t term_first, term_count;  // levels added to layer j + 1
};
__global__ void __launch_bounds__(FRI_TAIL_BLOCK) k_fri_tail(const FriRound* rounds, uint32_t n_rounds, uint32_t j0,
                                                   const AxpyTerm* terms, const uint32_t* pre, uint32_t* chal,
                                                   uint32_t inv2) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(FRI_TAIL_BLOCK / 32)];
  __shared__ uint32_t msg[64];
  p2_load_full_keys(keys);  // ends with a barrier
  P2Lane L;
  L.init(keys);
  const uint32_t per = (blockDim.x >> 5) * P2_GROUPS_PER_WARP;
  const uint32_t first = (threadIdx.x >> 5) * P2_GROUPS_PER_WARP, group = (uint32_t)L.base / 6;
  for (uint32_t r = 0; r < n_rounds; r++) {
    const FriRound R = rounds[r];
    const uint32_t j = j0 + r;
    const uint64_t half = R.n / 2;
    // fold
    {
      E6 alpha;
#pragma unroll
      for (int w = 0; w < 6; w++) alpha.c[w] = chal[8 * (size_t)j + w];
      int lg = 0;
      while ((1ull << lg) < half) lg++;
      for (uint64_t i = threadIdx.x; i < half; i += blockDim.x) {
        const uint32_t e = bitrev32((uint32_t)i, lg);
        const uint32_t xinv = __ldg(R.tw + ((R.n - e) & (R.n - 1)));
        const E6 p = ld6(R.cur, R.n, 2 * i), q = ld6(R.cur, R.n, 2 * i + 1);
        const E6 sm = e6_mul_base(e6_add(p, q), inv2);
        const E6 d = e6_mul(e6_mul_base(e6_mul_base(e6_sub(p, q), inv2), xinv), alpha);
        E6 v = e6_add(sm, d);
        for (uint32_t t = 0; t < R.term_count; t++) {
          const AxpyTerm T = terms[R.term_first + t];
          v = e6_add(v, e6_mul(ld6(T.lvl, half, i), ld_e6w(T.gamma)));
        }
        st6(R.next, half, i, v);
      }
    }
    __syncthreads();
    if (!R.nodes) break;
    // leaves of layer j + 1: Sponge(LEAF, 0, 2, row 2k, row 2k + 1), 15 elements
    const uint32_t nl = 1u << R.log_leaves;
    {
      LeafGroup g;
      g.base = nullptr;
      g.ext = R.next;
      g.stride = half;
      g.nb = 0;
      g.ne = 1;
      g.n_leaves = nl;
      g.out = R.nodes + (size_t)8 * nl;
      const uint32_t h0 = to_mont(LEAF_TAG), h1 = to_mont(0), h2 = to_mont(2);
      for (uint32_t k0 = first; k0 < nl; k0 += per) {
        const uint32_t k = k0 + group;
        const bool active = L.lane < 30 && k < nl;
        uint32_t x[4] = {0, 0, 0, 0};
        if (active && L.idx < 4) {
#pragma unroll
          for (uint32_t i = 0; i < 4; i++) {
            const uint32_t e = 4 * L.idx + i;
            if (e < 15) x[i] = leaf_elem(g, e, k, h0, h1, h2);
          }
        }
        p2c_permute(x, L, keys);
        if (active && L.idx < 2) {
          uint32_t* o = g.out + (size_t)k * 8 + 4 * L.idx;
#pragma unroll
          for (int i = 0; i < 4; i++) o[i] = x[i];
        }
      }
    }
    __syncthreads();
    for (uint32_t w = nl >> 1; w >= 1; w >>= 1) {
      for (uint32_t i0 = first; i0 < w; i0 += per) {
        const uint32_t i = i0 + group;
        merkle_node(R.nodes, (uint64_t)w + i, L, keys, L.lane < 30 && i < w);
      }
      __syncthreads();
    }
    // challenge j + 1 = sponge(name elements || challenge j || root)
    const uint32_t total = R.pre_len + 16;
    for (uint32_t i = threadIdx.x; i < total; i += blockDim.x)
      msg[i] = i < R.pre_len ? pre[R.pre_off + i] : (i < R.pre_len + 8 ? chal[8 * (size_t)j + (i - R.pre_len)]
                                                                          : R.nodes[8 + (i - R.pre_len - 8)]);
    __syncthreads();
    if (threadIdx.x < 32) {
      uint32_t x[4] = {0, 0, 0, 0};
      for (uint32_t b = 0; b < total; b += 16) {
        const uint32_t len = min(16u, total - b);
        if (L.idx < 4)
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (4 * (uint32_t)L.idx + k < len) x[k] = msg[b + 4 * L.idx + k];
        p2c_permute(x, L, keys);
      }
      if (L.lane < 2)
#pragma unroll
        for (int k = 0; k < 4; k++) chal[8 * (size_t)(j + 1) + 4 * L.lane + k] = x[k];
    }
    __syncthreads();
  }
}

// One Fiat-Shamir challenge on the device, for challenges whose bindings are
// already in device memory (the FRI layer roots): digest = state[0..8) of
// the width-24 sponge (rate 16, overwrite, no padding) over
// pre[0..n_pre) || prev[0..8) || bind[0..8), as Transcript::compute on the
// host (internal/fiat-shamir/transcript.go:221-315).  One warp, six lanes
// per permutation; `out` gets 8 words.
__global__ void k_fs_challenge(const uint32_t* pre, uint32_t n_pre, const uint32_t* prev, const uint32_t* bind,
                               uint32_t* out) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(1)];
  __shared__ uint32_t msg[64];
  const uint32_t total = n_pre + 16;  // n_pre <= 48, checked by the host
  for (uint32_t i = threadIdx.x; i < total; i += blockDim.x)
    msg[i] = i < n_pre ? pre[i] : (i < n_pre + 8 ? prev[i - n_pre] : bind[i - n_pre - 8]);
  p2_load_full_keys(keys);  // ends with a barrier
  P2Lane L;
  L.init(keys);
  uint32_t x[4] = {0, 0, 0, 0};
  for (uint32_t b = 0; b < total; b += 16) {
    const uint32_t len = min(16u, total - b);  // words 0..len of the state are overwritten
    if (L.idx < 4)
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (4 * (uint32_t)L.idx + k < len) x[k] = msg[b + 4 * L.idx + k];
    p2c_permute(x, L, keys);
  }
  if (L.lane < 2)
#pragma unroll
    for (int k = 0; k < 4; k++) out[4 * L.lane + k] = x[k];
}

// A chain of Fiat-Shamir challenges on the device, computed in order:
// challenge i hashes msg[moff, moff + total) as k_fs_challenge does and
// writes its 8 digest words to `out`.  The message words come from segments
// — host constants uploaded with the descriptors (names' elements, known
// bindings) and words already in device memory (roots, exposed values, the
// digest of a challenge computed by an earlier launch) — all read up front,
// one segment per thread at a time; a digest that the next challenge of the
// same chain hashes is forwarded from registers to msg[fwd] instead.  One
// warp, six lanes per permutation; the chain's messages hold at most
// FS_MAX_MSG words (checked by the host).
constexpr uint32_t FS_MAX_MSG = 4096;
struct FsSeg { const uint32_t* src; uint32_t len, off; };
struct FsChal { uint32_t moff, total; uint32_t* out; int32_t fwd; };
__global__ void __launch_bounds__(32) k_fs_chain(const FsChal* chals, uint32_t n_chals, const FsSeg* segs,
                                                 uint32_t n_segs) {
  __shared__ __align__(16) uint32_t keys[p2c_smem_words(1)];
  __shared__ uint32_t msg[FS_MAX_MSG];
  for (uint32_t s = threadIdx.x; s < n_segs; s += blockDim.x) {
    const FsSeg sg = segs[s];
    for (uint32_t k = 0; k < sg.len; k++) msg[sg.off + k] = sg.src[k];
  }
  p2_load_full_keys(keys);  // ends with a barrier
  P2Lane L;
  L.init(keys);
  for (uint32_t i = 0; i < n_chals; i++) {
    const FsChal ch = chals[i];
    uint32_t x[4] = {0, 0, 0, 0};
    for (uint32_t b = 0; b < ch.total; b += 16) {
      const uint32_t len = min(16u, ch.total - b);  // words 0..len of the state are overwritten
      if (L.idx < 4)
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (4 * (uint32_t)L.idx + k < len) x[k] = msg[ch.moff + b + 4 * L.idx + k];
      p2c_permute(x, L, keys);
    }
    if (L.lane < 2)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        ch.out[4 * L.lane + k] = x[k];
        if (ch.fwd >= 0) msg[ch.fwd + 4 * L.lane + k] = x[k];
      }
    __syncwarp();
  }
}

// The challenge table of the step and quotient kernels: the round coins (the
// first six words of each digest slot, slot stride 8), then the exposed
// values times ninv[e] (1/n of the producing module; 0 while entry e is not
// produced yet, which zeroes it) and the exposed values themselves.
__global__ void k_coins_assemble(const uint32_t* slots, uint32_t n_coins, const uint32_t* exposed,
                                 const uint32_t* ninv, uint32_t n_exp, uint32_t* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t nc = 6 * n_coins, ne = 6 * n_exp;
  if (i < nc) {
    out[i] = slots[8 * (i / 6) + i % 6];
  } else if (i < nc + ne) {
    const uint32_t k = i - nc, f = ninv[k / 6];
    out[i] = f ? mul(exposed[k], f) : 0u;
  } else if (i < nc + 2 * ne) {
    const uint32_t k = i - nc - ne;
    out[i] = ninv[k / 6] ? exposed[k] : 0u;
  }
}

// ---------------------------------------------------------------- openings
// A Montgomery word in the proof encoding: canonical, big-endian bytes.
__device__ __forceinline__ uint32_t proof_word(uint32_t m) { return __byte_perm(from_mont(m), 0, 0x0123); }

// Row pairs: for every query q and source, the rows lo and lo + 1 of each
// lane, lo = (s_q >> shift) & ~1: row lo of every lane, then row lo + 1, at
// out[q * per_q + off + h * n_lanes + lane] (the order the proof lists them).
struct RowSrc { const uint32_t* lane0; uint64_t lane_stride; uint32_t n_lanes; uint32_t shift; uint64_t off; };
__global__ void k_gather_rows(const RowSrc* srcs, uint32_t n_src, const uint32_t* pos, uint32_t nq, uint64_t per_q,
                              uint32_t* out) {
  const uint32_t q = blockIdx.y;
  const RowSrc s = srcs[blockIdx.z];
  const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq || l >= s.n_lanes) return;
  uint32_t lo = (pos[q] >> s.shift) & ~1u;
  const uint32_t* p = s.lane0 + l * s.lane_stride;
  out[q * per_q + s.off + l] = proof_word(p[lo]);
  out[q * per_q + s.off + s.n_lanes + l] = proof_word(p[lo + 1]);
}

// Merkle paths: siblings of leaf idx = ((s_q >> shift) >> 1), leaf level
// first, then the injection leaves inj_t[idx >> d_t].
struct PathSrc {
  const uint32_t* nodes;
  const uint32_t* const* inj;
  const uint32_t* inj_shift;  // d_t = log2(n_leaves / width_t)
  uint32_t log_leaves;
  uint32_t n_inj;
  uint32_t shift;
  uint64_t off;
};
__global__ void k_gather_paths(const PathSrc* srcs, const uint32_t* pos, uint32_t nq, uint64_t per_q, uint32_t* out) {
  const uint32_t q = blockIdx.y;
  const PathSrc s = srcs[blockIdx.z];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq || t >= s.log_leaves + s.n_inj) return;
  uint32_t idx = (pos[q] >> s.shift) >> 1;
  uint32_t* o = out + q * per_q + s.off + (uint64_t)t * 8;
  const uint32_t* src;
  if (t < s.log_leaves) {
    uint64_t node = (((uint64_t)1 << s.log_leaves) + idx) >> t;
    src = s.nodes + (node ^ 1) * 8;
  } else {
    uint32_t k = t - s.log_leaves;
    src = s.inj[k] + (uint64_t)(idx >> s.inj_shift[k]) * 8;
  }
  for (int w = 0; w < 8; w++) o[w] = proof_word(src[w]);
}

// Per-query proof sections.  Every query's part of a section has the same
// layout, described once per section by a word map: code >> 30 = 0 copies
// gathered word (code & 0x3fffffff) of the query, 1 is constant word
// consts[code & ..], 2 is a position word of pos_ops[code & ..] (the query's
// row or leaf index at some layer).  Output: big-endian words, query k of
// section s at out + s.out_off + k * s.q_words.
struct PosOp { uint32_t shift, leaf; };
struct SectionSrc { uint64_t map_off, out_off; uint32_t q_words; };
constexpr uint32_t SEC_COPY = 0u, SEC_CONST = 1u, SEC_POS = 2u;
__global__ void k_assemble(const SectionSrc* secs, const uint32_t* map, const uint32_t* consts, const PosOp* pops,
                           const uint32_t* pos, const uint32_t* gathered, uint64_t per_q, uint32_t nq, uint32_t* out) {
  const SectionSrc sc = secs[blockIdx.z];
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (j >= sc.q_words || k >= nq) return;
  const uint32_t code = map[sc.map_off + j], kind = code >> 30, idx = code & 0x3fffffffu;
  uint32_t w;
  if (kind == SEC_COPY) {
    w = gathered[(uint64_t)k * per_q + idx];  // already encoded (proof_word)
  } else {
    uint32_t v;
    if (kind == SEC_CONST) {
      v = consts[idx];
    } else {
      const PosOp op = pops[idx];
      v = pos[k] >> op.shift;
      if (op.leaf) v = (v & ~1u) >> 1;
    }
    w = __byte_perm(v, 0, 0x0123);
  }
  out[sc.out_off + (uint64_t)k * sc.q_words + j] = w;
  // the section's query count stands before it, as in the proof
  if (j == 0 && k == 0) out[sc.out_off - 1] = __byte_perm(nq, 0, 0x0123);
}

}  // namespace lg
