// Scans over E6 values: products (grand products, running ratios) or sums
// (logup running sums), and the grand product of rows as callers hold them
// (ext.E6 arrays, six words a row).  Everything here multiplies exactly, so
// the order of the factors does not show in the results.
#pragma once
#include <type_traits>

#include "field.cuh"

namespace lg {

template <bool SUM> __device__ __forceinline__ E6 scan_id() { return SUM ? e6_zero() : e6_one(); }
template <bool SUM> __device__ __forceinline__ E6 scan_op(const E6& a, const E6& b) {
  return SUM ? e6_add(a, b) : e6_mul(a, b);
}
__device__ __forceinline__ E6 e6_shfl_up(const E6& v, int d) {
  E6 r;
#pragma unroll
  for (int w = 0; w < 6; w++) r.c[w] = __shfl_up_sync(0xffffffffu, v.c[w], d);
  return r;
}

// Exclusive scan of one value per thread over a block of T threads (a power
// of two of whole warps, at most 32 of them): within warps by shuffles, then
// over the warps' totals in the first warp.  `total` (every thread): the
// block's.  Two barriers; `sh` holds T/32 values.
template <bool SUM, int T> __device__ __forceinline__ E6 block_scan(E6 v, E6* sh, E6& total) {
  constexpr int W = T / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int d = 1; d < 32; d <<= 1) {
    const E6 t = e6_shfl_up(v, d);
    if (lane >= d) v = scan_op<SUM>(t, v);
  }
  if (lane == 31) sh[warp] = v;
  __syncthreads();
  if (W > 1 && warp == 0) {
    E6 a = lane < W ? sh[lane] : scan_id<SUM>();
#pragma unroll 1
    for (int d = 1; d < W; d <<= 1) {
      const E6 t = e6_shfl_up(a, d);
      if (lane >= d) a = scan_op<SUM>(t, a);
    }
    if (lane < W) sh[lane] = a;
  }
  __syncthreads();
  total = sh[W - 1];
  const E6 before = e6_shfl_up(v, 1);
  E6 pre = lane ? before : scan_id<SUM>();
  if (warp) pre = scan_op<SUM>(sh[warp - 1], pre);
  return pre;
}

// ---------------------------------------------------------------- rows
// VEC: the rows are aligned to 8 bytes (three 8-byte accesses a row).
template <bool VEC> __device__ __forceinline__ E6 ld_row(const uint32_t* p, uint64_t i) {
  E6 r;
  if constexpr (VEC) {
    const uint2* q = reinterpret_cast<const uint2*>(p + 6 * i);
    const uint2 a = q[0], b = q[1], c = q[2];
    r = E6{{a.x, a.y, b.x, b.y, c.x, c.y}};
  } else {
#pragma unroll
    for (int w = 0; w < 6; w++) r.c[w] = p[6 * i + w];
  }
  return r;
}
template <bool VEC> __device__ __forceinline__ void st_row(uint32_t* p, uint64_t i, const E6& v) {
  if constexpr (VEC) {
    uint2* q = reinterpret_cast<uint2*>(p + 6 * i);
    q[0] = make_uint2(v.c[0], v.c[1]);
    q[1] = make_uint2(v.c[2], v.c[3]);
    q[2] = make_uint2(v.c[4], v.c[5]);
  } else {
#pragma unroll
    for (int w = 0; w < 6; w++) p[6 * i + w] = v.c[w];
  }
}
__device__ __forceinline__ bool e6_is_zero(const E6& v) {
  return (v.c[0] | v.c[1] | v.c[2] | v.c[3] | v.c[4] | v.c[5]) == 0;
}

// Tile shapes of the row kernels: T threads of R consecutive rows.  A thread's
// rows share one inversion, so long inputs take R = 8; short ones take fewer
// rows a thread so that the tiles reach every SM (148 of them on B200).
constexpr uint32_t GP_TILE_S = 128, GP_TILE_M = 512, GP_TILE_L = 2048;
inline uint32_t gp_tile(uint64_t n) { return n <= 1u << 16 ? GP_TILE_S : n <= 1u << 18 ? GP_TILE_M : GP_TILE_L; }

// Exclusive product scan inside each tile of T R rows: of the ratios
// num / den (RATIO; x is written; a ratio is 0 where its denominator is 0, as
// e6_inv(0) = 0), or of x in place.  Tile t's product goes to totals[6 t + w].
// A tile's rows are read before any of them is written.
//
// With A_i = num_0 .. num_(i-1) and B_i = den_i .. den_(R-1) over a thread's
// rows, the product of the ratios before row i is A_i B_i / B_0: one inversion
// for all R rows and three E6 products a row, where an inversion takes about
// six.  The denominators are taken from the back and the numerators from the
// front, one row at a time, so only the products stay in registers.
// What bounds it: the integer-multiply pipe (about five E6 products a row; 61%
// of its peak) and, with 16 warps an SM, the loads' latency (long scoreboard 2.2
// per issue; a row's 24 B are fetched where they lie, L1 at 47%); for few tiles, the dependent products of the scan and the inversion.
// 512 threads an SM, 128 registers each: with both operands of every row held
// (210 registers) 1,000,003 rows took 162 us and not 127 (start to end; 98 with
// the extension products of one reduction per coefficient).
template <int T, int R, bool VEC, bool RATIO>
__global__ void __launch_bounds__(T, 512 / T) k_rows_scan(const uint32_t* num, const uint32_t* den, uint64_t n,
                                                          uint32_t* x, uint32_t* totals) {
  __shared__ E6 sh[T / 32];
  const uint64_t base = (uint64_t)blockIdx.x * (T * R) + (uint64_t)threadIdx.x * R;
  E6 v[R], acc;
  if constexpr (RATIO) {
    uint32_t zero = 0;  // rows whose denominator is 0
    E6 b = e6_one();
#pragma unroll
    for (int i = R - 1; i >= 0; i--) {
      E6 d = base + i < n ? ld_row<VEC>(den, base + i) : e6_one();
      if (e6_is_zero(d)) {
        zero |= 1u << i;
        d = e6_one();
      }
      b = i == R - 1 ? d : e6_mul(d, b);
      v[i] = b;
    }
    acc = e6_inv(b);
    v[0] = e6_one();
#pragma unroll
    for (int i = 0; i < R; i++) {
      if (i) v[i] = e6_mul(acc, v[i]);
      E6 a = base + i < n ? ld_row<VEC>(num, base + i) : e6_one();
      if (zero >> i & 1) a = e6_zero();
      acc = e6_mul(acc, a);
    }
  } else {
    acc = e6_one();
#pragma unroll
    for (int i = 0; i < R; i++) {
      v[i] = acc;
      if (base + i < n) acc = e6_mul(acc, ld_row<VEC>(x, base + i));
    }
  }
  E6 total;
  const E6 pre = block_scan<false, T>(acc, sh, total);
#pragma unroll
  for (int i = 0; i < R; i++)
    if (base + i < n) st_row<VEC>(x, base + i, e6_mul(v[i], pre));
  if (threadIdx.x < 6) totals[6 * (uint64_t)blockIdx.x + threadIdx.x] = total.c[threadIdx.x];
}

// x[i] *= the product of the tiles before tile i / tile.  PREFIX: `pre` holds
// those products; otherwise the totals, which every block multiplies up to its
// own tile (the tiles before it over T threads, at most four E6 products each,
// and the block's reduction), saving the launch between.
// The block's rows are loaded before that, so the two overlap.
template <int T, int R, bool VEC, bool PREFIX>
__global__ void __launch_bounds__(T, 512 / T) k_rows_apply(uint32_t* x, uint64_t n, const uint32_t* pre) {
  __shared__ E6 sh[T / 32];
  if (blockIdx.x == 0) return;  // nothing before the first tile
  const uint64_t first = (uint64_t)blockIdx.x * (T * R) + threadIdx.x;
  E6 v[R], p;
#pragma unroll
  for (int i = 0; i < R; i++)
    if (first + i * T < n) v[i] = ld_row<VEC>(x, first + i * T);
  if constexpr (PREFIX) {
    p = ld_row<true>(pre, blockIdx.x);
  } else {
    E6 acc = e6_one();
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += T) acc = e6_mul(acc, ld_row<true>(pre, t));
    block_scan<false, T>(acc, sh, p);
  }
#pragma unroll
  for (int i = 0; i < R; i++)
    if (first + i * T < n) st_row<VEC>(x, first + i * T, e6_mul(v[i], p));
}

// Exclusive prefix products of nt tile totals, one block of T threads.
template <int T> __global__ void __launch_bounds__(T) k_rows_prefix(const uint32_t* totals, uint32_t nt, uint32_t* pre) {
  __shared__ E6 sh[T / 32];
  const uint32_t per = (nt + T - 1) / T, first = threadIdx.x * per;
  E6 acc = e6_one();
  for (uint32_t i = 0; i < per && first + i < nt; i++) acc = e6_mul(acc, ld_row<true>(totals, first + i));
  E6 total;
  acc = block_scan<false, T>(acc, sh, total);
  for (uint32_t i = 0; i < per && first + i < nt; i++) {
    st_row<true>(pre, first + i, acc);
    acc = e6_mul(acc, ld_row<true>(totals, first + i));
  }
}

// Element-wise ratios, R rows per thread.
template <int T, int R, bool VEC>
__global__ void __launch_bounds__(T) k_rows_ratio(const uint32_t* num, const uint32_t* den, uint64_t n, uint32_t* out) {
  const uint64_t base = ((uint64_t)blockIdx.x * T + threadIdx.x) * R;
  E6 a[R], d[R], b[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    const bool in = base + i < n;
    a[i] = in ? ld_row<VEC>(num, base + i) : e6_one();
    d[i] = in ? ld_row<VEC>(den, base + i) : e6_one();
    if (e6_is_zero(d[i])) {
      a[i] = e6_zero();
      d[i] = e6_one();
    }
    b[i] = i ? e6_mul(b[i - 1], d[i]) : d[0];
  }
  E6 inv = e6_inv(b[R - 1]);  // 1 / (d_0 .. d_i), from the back
#pragma unroll
  for (int i = R - 1; i >= 0; i--) {
    const E6 q = e6_mul(a[i], i ? e6_mul(inv, b[i - 1]) : inv);
    if (i) inv = e6_mul(inv, d[i]);
    if (base + i < n) st_row<VEC>(out, base + i, q);
  }
}

// Calls f(T, R) as integral constants for the tile shape of n rows.
template <class F> inline void with_gp_shape(uint64_t n, F&& f) {
  switch (gp_tile(n)) {
    case GP_TILE_S: f(std::integral_constant<int, 128>{}, std::integral_constant<int, 1>{}); break;
    case GP_TILE_M: f(std::integral_constant<int, 128>{}, std::integral_constant<int, 4>{}); break;
    default: f(std::integral_constant<int, 256>{}, std::integral_constant<int, 8>{}); break;
  }
}

}  // namespace lg
