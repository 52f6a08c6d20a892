// Grand product without any device allocation: lg_grand_product_noalloc.
//
// Who needs it: callers that cannot call cudaMalloc — code running where a
// caching allocator owns the device memory and forbids raw allocations, code
// inside a memory-capped sandbox, or a host that must not add allocation
// latency to its request path.  They pass inputs and outputs they already
// own; the only scratch this entry point uses is the file-scope device array
// below (the tile totals and their prefix products), which every GPU that
// loads this library holds until the process exits.
//
// Same result as lg_grand_product: out[0] = 1, out[i] = prod_{k<i} num[k]/den[k].
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/loom_gpu.h"
#include "scan.cuh"

namespace lg {
// Kernel launch counter of the library (lg_kernel_launches), defined with the
// other entry points.
void note_launches(uint64_t k);
}  // namespace lg

namespace {

using namespace lg;

constexpr uint64_t NOALLOC_GP_MAX_ROWS = 1ull << 22;  // the largest loom module (2^22 rows)
constexpr uint32_t NA_MAX_TILES = (uint32_t)(NOALLOC_GP_MAX_ROWS / GP_TILE_L);  // 2048
static_assert((1u << 16) / GP_TILE_S <= NA_MAX_TILES && (1u << 18) / GP_TILE_M <= NA_MAX_TILES, "tiles fit the scratch");

// Tile totals [0, 6 * NA_MAX_TILES) and their exclusive prefix products
// [6 * NA_MAX_TILES, 12 * NA_MAX_TILES): 96 KiB.  Every word a call reads is
// written earlier in the same call, so nothing has to be cleared.
static __device__ __align__(256) uint32_t g_gp_scratch[12 * NA_MAX_TILES];

// Device address of g_gp_scratch, looked up once per device with that
// device current (host code cannot use the symbol's name as a pointer).
std::mutex g_mu;
constexpr int MAX_DEVICES = 64;
uint32_t* g_scratch_ptr[MAX_DEVICES] = {};

int scratch_for_current_device(uint32_t** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return LG_ERR_CUDA;
  if (dev < 0 || dev >= MAX_DEVICES) return LG_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_gp_scratch) != cudaSuccess || !p) return LG_ERR_CUDA;
    g_scratch_ptr[dev] = (uint32_t*)p;
  }
  *out = g_scratch_ptr[dev];
  return LG_OK;
}

}  // namespace

extern "C" int lg_grand_product_noalloc(const uint32_t* num, const uint32_t* den, uint64_t n, uint32_t* out,
                                        void* stream) {
  if (!num || !den || !out || n == 0) return LG_ERR_INVALID;
  if (n > NOALLOC_GP_MAX_ROWS) return LG_ERR_UNSUPPORTED;
  // An error already pending on this thread (from the caller's own work) is
  // left in place and reported, not cleared and taken for one of ours.
  if (cudaPeekAtLastError() != cudaSuccess) return LG_ERR_CUDA;
  uint32_t* scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc != LG_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const uint32_t tile = gp_tile(n), nt = (uint32_t)((n + tile - 1) / tile);
  uint32_t* totals = scratch;
  uint32_t* pre = scratch + 6 * NA_MAX_TILES;
  with_gp_shape(n, [&](auto TC, auto RC) {
    constexpr int T = decltype(TC)::value, R = decltype(RC)::value;
    auto go = [&](auto V) {
      constexpr bool VEC = decltype(V)::value;
      k_rows_ratio<T, R, VEC><<<nt, T, 0, st>>>(num, den, n, out);
      k_rows_scan<T, R, VEC, false><<<nt, T, 0, st>>>(nullptr, nullptr, n, out, totals);
      k_rows_prefix<256><<<1, 256, 0, st>>>(totals, nt, pre);
      k_rows_apply<T, R, VEC, true><<<nt, T, 0, st>>>(out, n, pre);
    };
    if (((uintptr_t)num | (uintptr_t)den | (uintptr_t)out) & 7) go(std::false_type{});
    else go(std::true_type{});
  });
  note_launches(4);
  return cudaGetLastError() == cudaSuccess ? LG_OK : LG_ERR_CUDA;
}
