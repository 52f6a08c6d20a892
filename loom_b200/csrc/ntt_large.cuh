// Transforms of 2^15 .. 2^22 points: four-step, two passes through a scratch
// buffer (inverse transforms and the quotient's cosets; the coset transforms of
// an LDE take the forward tree further down).  With n = R C (R = 2^floor(log n / 2), C = 2^ceil(log n / 2)),
// k = k1 + R k2 and j = C j1 + j2:
//   X[C j1 + j2] = sum_k1 w_R^(j1 k1) w_n^(j2 k1) sum_k2 w_C^(j2 k2) x[k1 + R k2].
// Pass A: for a tile of 16 consecutive k1, the length-C transforms over k2
// (the tile's 16 columns are read 64 bytes at a time), times w_n^(j2 k1), into
// scratch[j2 R + k1].  Pass B: for a tile of 16 consecutive j2, the length-R
// transforms over k1 (scratch rows, contiguous), stored in natural order.
// Input scaling x[k] * c0 * t1[k] * t2[(e k) mod m2] covers 1/n
// and the coset shifts.
//
// The 16 sub-transforms of a tile run together in shared memory with the
// radix-16 register passes of ntt16.cuh (16 elements of one column per thread,
// four stages per shared-memory round trip), the columns interleaved: element
// (row, col) at 16 (row + row / 16) + (col ^ (row mod 16)).  The row padding
// keeps the two half-warps of a pass in different banks, the column swizzle
// keeps the row-wise staging of pass B conflict-free.
#pragma once
#include "kernels.cuh"

namespace lg {

constexpr int BIG_TILE = 16;

struct BigNtt {
  const uint32_t* in;
  uint32_t* out;
  uint32_t* scratch;       // n words
  const uint32_t* t1;      // optional table of n words (Montgomery)
  const uint32_t* t2;      // optional: the coset shift w_4n^((e2 k) mod 4n) (set: the w_4n table)
  uint32_t m2_mask, e2;    // t2 index = (e2 * k) & m2_mask
  uint32_t c0;             // constant factor (Montgomery)
  uint32_t c0c, c0s;       // c0 canonical and its Shoup companion (big_ntt sets them)
  uint32_t* coset0;        // pass A also writes its input in bit-reversed order here (16-byte aligned; null: no)
};

__device__ __forceinline__ uint32_t tile_addr(uint32_t row, uint32_t col) {
  return ((row + (row >> 4)) << 4) + (col ^ (row & 15u));
}
// words of one tile of 16 columns of 2^logl rows
__host__ __device__ constexpr size_t tile_words(int logl) {
  return (((size_t)1 << logl) + ((size_t)1 << logl) / 16) * 16;
}

// The 16 column transforms of a tile, 2^LOGL rows each (`tw`: the tw16
// tables of 2^LOGL points).  Pass 0 takes its
// inputs from first(col, row) (global memory, or the staged tile), every pass
// but the last writes back to S, the last hands each element to
// store(col, row, value).  DIF: natural rows in, bit-reversed rows out.
struct NoTileHook {
  __device__ void operator()(uint32_t, uint32_t, int, uint32_t*) const {}
};
// `loaded(col, t, lo, v)` sees a thread's 16 inputs of pass 0 before its
// butterflies and may change them.
template <bool DIF, int LOGL, class First, class Store, class Loaded = NoTileHook>
__device__ __forceinline__ void ntt16_tile(uint32_t* S, const uint32_t* tw, bool inverse, First first, Store store,
                                           Loaded loaded = Loaded()) {
  constexpr uint32_t groups = (1u << LOGL) >> 4;  // per column
  constexpr int np = (LOGL - ((LOGL & 3) ? (LOGL & 3) : 4)) / 4 + 1;
  constexpr uint32_t comp = tw16_words(LOGL);
#pragma unroll
  for (int p = 0; p < np; p++) {
    int lo = 0, s_lo = 0, s_hi = 0;
    pass_plan<DIF>(p, LOGL, lo, s_lo, s_hi);
    const uint32_t* ptab = tw + tw16_pass_offset(LOGL, DIF, inverse, p);
    for (uint32_t u = threadIdx.x; u < groups * BIG_TILE; u += blockDim.x) {
      const uint32_t col = u & (BIG_TILE - 1), t = u >> 4;
      uint32_t v[16];
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t row = grp_index(t, r, lo);
        v[r] = p == 0 ? first(col, row) : S[tile_addr(row, col)];
      }
      if (p == 0) loaded(col, t, lo, v);
      pass16<DIF>(v, t, lo, s_lo, s_hi, ptab, comp, inverse);
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t row = grp_index(t, r, lo);
        if (p == np - 1) store(col, row, v[r]);
        else S[tile_addr(row, col)] = v[r];
      }
    }
    __syncthreads();
  }
}

// A product v w^e by a power of a root w of order 2^(11 + k), from two small
// tables that stay in L1: lo[i] = w^i (i < 2^11) and hi[i] = w^(2^11 i), each
// entry a canonical word with its Shoup companion (Ctx::split_powers): two
// Shoup products instead of a table product and a Montgomery product.
constexpr int TW_SPLIT = 11;
__device__ __forceinline__ uint32_t mul_split(uint32_t v, const uint2* tab, uint32_t e) {
  const uint2 a = __ldg(tab + (e & ((1u << TW_SPLIT) - 1))), b = __ldg(tab + (1u << TW_SPLIT) + (e >> TW_SPLIT));
  return mulc(mulc_lazy(v, a.x, a.y), b.x, b.y);
}

// tw_n: w_n split (mul_split layout); t2s: the same for w_4n (the coset
// shifts); tw_c: the tw16 tables of C points.  Block (x, y): tile x of job y.
template <int LOGC>
__global__ void __launch_bounds__(512, 2) k_big_pass_a(const BigNtt* jobs, int logn, int logr, int inverse,
                                                    const uint2* tw_n, const uint2* t2s, const uint32_t* tw_c) {
  extern __shared__ uint32_t S[];
  const BigNtt J = jobs[blockIdx.y];
  const uint32_t R = 1u << logr, n = 1u << logn;
  const uint32_t k1_0 = blockIdx.x * BIG_TILE;
  auto first = [&](uint32_t col, uint32_t k2) { return J.in[(k1_0 + col) + R * k2]; };
  auto loaded = [&](uint32_t col, uint32_t t, int lo, uint32_t* v) {
    if (J.coset0) {
      // k = k1 + R k2 goes to bitrev(k1) C + bitrev(k2): the thread's rows
      // k2 = t + r C/16 are 16 consecutive words in the order bitrev(r)
      uint4* q = reinterpret_cast<uint4*>(J.coset0 + ((size_t)bitrev32(k1_0 + col, logr) << LOGC) +
                                          (bitrev32(t, LOGC - 4) << 4));
      q[0] = make_uint4(v[0], v[8], v[4], v[12]);
      q[1] = make_uint4(v[2], v[10], v[6], v[14]);
      q[2] = make_uint4(v[1], v[9], v[5], v[13]);
      q[3] = make_uint4(v[3], v[11], v[7], v[15]);
    }
#pragma unroll
    for (uint32_t r = 0; r < 16; r++) {
      const uint32_t k = (k1_0 + col) + R * grp_index(t, r, lo);
      if (J.c0 != MONT_ONE) v[r] = mulc(v[r], J.c0c, J.c0s);
      if (J.t1) v[r] = mul(v[r], __ldg(J.t1 + k));
      if (J.t2) v[r] = mul_split(v[r], t2s, (J.e2 * k) & J.m2_mask);
    }
  };
  auto store = [&](uint32_t col, uint32_t p, uint32_t v) {
    const uint32_t j2 = bitrev32(p, LOGC), k1 = k1_0 + col;
    uint32_t e = (uint32_t)(((uint64_t)j2 * k1) & (n - 1));
    if (inverse) e = (n - e) & (n - 1);
    J.scratch[(uint64_t)j2 * R + k1] = mul_split(v, tw_n, e);
  };
  ntt16_tile<true, LOGC>(S, tw_c, inverse != 0, first, store, loaded);
}

// Block (x, y): rows [16 x, 16 x + 16) of job y's scratch.
template <int LOGR>
__global__ void __launch_bounds__(512, 2) k_big_pass_b(const BigNtt* jobs, int logc, int inverse,
                                                    const uint32_t* tw_r) {
  extern __shared__ uint32_t S[];
  const BigNtt J = jobs[blockIdx.y];
  constexpr uint32_t R = 1u << LOGR;
  const uint32_t C = 1u << logc;
  const uint32_t j2_0 = blockIdx.x * BIG_TILE;
  // stage the 16 scratch rows (contiguous, coalesced) into the tile, every
  // copy in flight before the first wait
  for (uint32_t idx = threadIdx.x; idx < R * BIG_TILE; idx += blockDim.x) {
    const uint32_t jl = idx / R, k1 = idx % R;
    cp_async4(&S[tile_addr(k1, jl)], J.scratch + (uint64_t)(j2_0 + jl) * R + k1);
  }
  cp_async_wait_all();
  __syncthreads();
  auto first = [&](uint32_t col, uint32_t k1) { return S[tile_addr(k1, col)]; };
  auto store = [&](uint32_t col, uint32_t q, uint32_t v) {
    J.out[(uint64_t)C * bitrev32(q, LOGR) + j2_0 + col] = v;
  };
  ntt16_tile<true, LOGR>(S, tw_r, inverse != 0, first, store);
}

// ---------------------------------------------------------------- forward tree
// The coset transforms of a rate-4 LDE, coefficients in natural order to
// bit-reversed evaluations, as the lower part of one tree over the 4n points
// of <w_4n>: a node at depth D with index B stands for the polynomial modulo
// x^m - z, and its butterflies are (u + v w, u - v w) with the single twiddle
//   tau[B] = w_(2^(D+1))^bitrev_D(B),
// which does not depend on D.  Coset a is the subtree of node a at depth 2, so
// neither the coset's shift nor the twiddles between the two passes are
// products of their own, as they are in the four-step form (two table
// products each): pass A runs the depths below the coset's node on columns
// (stride R), pass B the remaining ones on rows of R consecutive words, in
// place in the output.  One table of tau (with Shoup companions) serves every
// size and coset.
//
// What bounds it: pass A the integer pipes (eight instructions a butterfly:
// multiply 58%, ALU 61%, issue 63% of their peaks), pass B the L1 data pipe
// (76%: the words' passes through shared memory and 120 B of twiddles per 16
// words of one column).  Per element of a 2^18-point transform the four-step
// form took 118 + 75 instructions, the tree 73 + 47.  Rate-4 encoding of 128
// columns of 2^18 rows on B200: 976 us, 1478 us with four-step coset transforms
// (a fourth of them for coset 0, which pass A of the inverse transform now
// writes as it reads the values).
struct FwdJob { const uint32_t* in; uint32_t* out; uint32_t node; };  // node: the coset a

// The first `levels` levels under node N on 16 registers (a group's elements,
// the distance halving from 8).  The twiddles of level k, tau[2^k N] ..
// tau[2^k N + 2^k - 1], are consecutive.
__device__ __forceinline__ void tree16(uint32_t v[16], const uint2* __restrict__ tau, uint32_t N, int levels) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (k >= levels) break;
    const uint32_t m = 1u << k, half = 8u >> k;  // m twiddles, butterflies at distance `half`
    uint32_t w[8], ws[8];
    const uint2* at = tau + ((size_t)N << k);
    if (k == 0) {
      const uint2 x = __ldg(at);
      w[0] = x.x;
      ws[0] = x.y;
    } else {
#pragma unroll
      for (uint32_t j = 0; j < m; j += 2) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(at + j));
        w[j] = x.x;
        ws[j] = x.y;
        w[j + 1] = x.z;
        ws[j + 1] = x.w;
      }
    }
#pragma unroll
    for (uint32_t j = 0; j < m; j++)
#pragma unroll
      for (uint32_t i = 0; i < half; i++) {
        uint32_t& a = v[j * 2 * half + i];
        uint32_t& b = v[j * 2 * half + half + i];
        const uint32_t u = a, x = mulc(b, w[j], ws[j]);
        a = add(u, x);
        b = sub(u, x);
      }
  }
}
// levels of pass p of a transform of 2^LOGL points: the DIF pass plan
LG_HD constexpr int tree_levels(int logl, int p) {
  const int rem = (logl & 3) ? (logl & 3) : 4;
  return p == 0 ? rem : 4;
}
LG_HD constexpr int tree_done(int logl, int p) {  // levels before pass p
  const int rem = (logl & 3) ? (logl & 3) : 4;
  return p == 0 ? 0 : rem + 4 * (p - 1);
}

// Pass A: block (x, y) the 16 columns from 16 x on of job y, 2^LOGC rows.
template <int LOGC>
__global__ void __launch_bounds__(512, 2) k_fwd_cols(const FwdJob* jobs, int logr, const uint2* __restrict__ tau) {
  extern __shared__ uint32_t S[];
  const FwdJob J = jobs[blockIdx.y];
  constexpr uint32_t groups = (1u << LOGC) >> 4;
  constexpr int np = pass_count(LOGC);
  const uint32_t k1_0 = blockIdx.x * BIG_TILE;
#pragma unroll
  for (int p = 0; p < np; p++) {
    const int lo = LOGC - tree_done(LOGC, p) - 4;
    for (uint32_t u = threadIdx.x; u < groups * BIG_TILE; u += blockDim.x) {
      const uint32_t col = u & (BIG_TILE - 1), t = u >> 4;
      uint32_t v[16];
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t row = grp_index(t, r, lo);
        v[r] = p == 0 ? __ldg(J.in + (((size_t)row << logr) + k1_0 + col)) : S[tile_addr(row, col)];
      }
      tree16(v, tau, (J.node << tree_done(LOGC, p)) + (t >> lo), tree_levels(LOGC, p));
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t row = grp_index(t, r, lo);
        if (p == np - 1) J.out[((size_t)row << logr) + k1_0 + col] = v[r];
        else S[tile_addr(row, col)] = v[r];
      }
    }
    if (p < np - 1) __syncthreads();
  }
}

// Pass B: 2^LOGR consecutive words per row, in place; block (x, y): the rows
// from x * FWD_ROWS(LOGR) on of job y.  A row's threads are consecutive.
constexpr int FWD_THREADS = 256;
LG_HD constexpr uint32_t fwd_rows(int logr) { return (uint32_t)FWD_THREADS * 16 >> logr; }
template <int LOGR>
__global__ void __launch_bounds__(FWD_THREADS, 4) k_fwd_rows(const FwdJob* jobs, int logc, const uint2* __restrict__ tau) {
  __shared__ uint32_t sm[FWD_THREADS * 17];
  const FwdJob J = jobs[blockIdx.y];
  constexpr uint32_t per = (1u << LOGR) >> 4;  // threads per row
  constexpr int np = pass_count(LOGR);
  const uint32_t t = threadIdx.x & (per - 1), rl = threadIdx.x / per;
  const uint32_t row = blockIdx.x * fwd_rows(LOGR) + rl;
  uint32_t* d = J.out + ((size_t)row << LOGR);
  uint32_t* S = sm + rl * per * 17;  // pad16 of the row's words
  const uint32_t node = (J.node << logc) + row;
  uint32_t v[16];
#pragma unroll
  for (int p = 0; p < np; p++) {
    const int lo = LOGR - tree_done(LOGR, p) - 4;
#pragma unroll
    for (uint32_t r = 0; r < 16; r++) v[r] = p == 0 ? d[grp_index(t, r, lo)] : S[pad16(grp_index(t, r, lo))];
    tree16(v, tau, (node << tree_done(LOGR, p)) + (t >> lo), tree_levels(LOGR, p));
    if (p == np - 1) {
      uint4* q = reinterpret_cast<uint4*>(d + 16 * t);
      q[0] = make_uint4(v[0], v[1], v[2], v[3]);
      q[1] = make_uint4(v[4], v[5], v[6], v[7]);
      q[2] = make_uint4(v[8], v[9], v[10], v[11]);
      q[3] = make_uint4(v[12], v[13], v[14], v[15]);
    } else {
      // a pass reads and writes the same words per thread, so one barrier
      // between passes is enough; rows of up to 512 words lie within a warp
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) S[pad16(grp_index(t, r, lo))] = v[r];
      if (per <= 32) __syncwarp();
      else __syncthreads();
    }
  }
}

// Calls f(std::integral_constant<int, L>{}) for the sub-transform sizes of
// the four-step path, 2^7 .. 2^11 rows.
template <class F> inline void with_tile_size(int logl, F&& f) {
  switch (logl) {
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 11: f(std::integral_constant<int, 11>{}); break;
    default: break;
  }
}

}  // namespace lg
