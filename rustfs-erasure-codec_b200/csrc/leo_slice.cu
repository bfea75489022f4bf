// leo_slice.cu -- launches of the bit-sliced Leopard GF(2^8) transforms
// (slice_fft.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "codec.hpp"
#include "launch_cfg.hpp"
#include "leo_slice.hpp"
#include "slice_fft.cuh"

namespace rsgpu {

#define RS_CUDA(expr)                              \
  do {                                             \
    cudaError_t e_ = (expr);                       \
    if (e_ != cudaSuccess) return cuda_status(e_); \
  } while (0)

namespace {

constexpr int kSliceMaxThreads = 1024;  // 64 registers

// Work item x of a launch: its job, the tile's first column and the job's
// shard length.
struct SliceItem {
  uint32_t job;
  uint64_t tile, len;
};
template <int WT>
__device__ __forceinline__ uint32_t slice_items(const SliceArgs &a) {
  return a.items ? a.n_items : uint32_t((a.len + 32 * WT - 1) / (32 * WT)) * a.n_jobs;
}
template <int WT>
__device__ __forceinline__ SliceItem slice_item(const SliceArgs &a, uint32_t x) {
  if (a.items) {
    const uint2 w = a.items[x];
    return SliceItem{w.x, uint64_t(w.y) * (32 * WT), a.lens[w.x]};
  }
  const uint32_t tiles_per_job = uint32_t((a.len + 32 * WT - 1) / (32 * WT)), job = x / tiles_per_job;
  return SliceItem{job, uint64_t(x - job * tiles_per_job) * (32 * WT), a.len};
}

template <int WT, bool VERIFY>
__global__ void __launch_bounds__(kSliceMaxThreads, 1) k_slice_encode(SliceArgs a) {
  extern __shared__ __align__(16) uint4 slice_smem[];
  const uint32_t total = slice_items<WT>(a);
#pragma unroll 1
  for (uint32_t x = blockIdx.x; x < total; x += gridDim.x) {
    const SliceItem it = slice_item<WT>(a, x);
    const LeoJob jd = a.jobs[it.job];
    const uint32_t bad = slice_encode_tile<WT, VERIFY>(uint32_t(__cvta_generic_to_shared(slice_smem)), a,
                                                       a.ptrs + jd.ptr_off, it.tile, it.len);
    if (VERIFY && __any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(a.flags + jd.flag_idx, 1u);
    __syncthreads();  // rows are free for the next tile
  }
}

template <int WT>
__global__ void __launch_bounds__(kSliceMaxThreads, 1) k_slice_decode(SliceArgs a) {
  extern __shared__ __align__(16) uint4 slice_smem[];
  __shared__ __align__(8) uint8_t need_bits[8];
  uint64_t *lane_ptrs = reinterpret_cast<uint64_t *>(slice_smem + size_t(a.n) * 2 * WT);
  const LaneInfo info{lane_ptrs, reinterpret_cast<uint8_t *>(lane_ptrs + a.n)};
  const uint32_t total = slice_items<WT>(a);
  uint32_t cur = ~0u;
#pragma unroll 1
  for (uint32_t x = blockIdx.x; x < total; x += gridDim.x) {
    const SliceItem it = slice_item<WT>(a, x);
    if (it.job != cur) {  // CTA-uniform; the rows and info are free (barrier below)
      cur = it.job;
      slice_lane_info(a, a.jobs[it.job], info, need_bits);
      __syncthreads();
    }
    slice_decode_tile<WT>(uint32_t(__cvta_generic_to_shared(slice_smem)), a, info, need_bits,
                          a.jobs[it.job].input_count, it.tile, it.len);
    __syncthreads();
  }
}

// Rows of a tile: decode n lanes; encode the accumulator and, with more than
// one data group, the scratch.
uint32_t slice_rows(int op, uint32_t k, uint32_t m, uint32_t n) {
  return op == RSGPU_OP_RECONSTRUCT ? n : (k > m ? 2 * m : m);
}

using SliceKernel = void (*)(SliceArgs);
SliceKernel slice_kernel(int op, uint32_t wt) {
  if (op == RSGPU_OP_RECONSTRUCT) return wt == 32 ? k_slice_decode<32> : k_slice_decode<28>;
  if (op == RSGPU_OP_VERIFY) return wt == 32 ? k_slice_encode<32, true> : k_slice_encode<28, true>;
  return wt == 32 ? k_slice_encode<32, false> : k_slice_encode<28, false>;
}

}  // namespace

namespace {
// Rows, threads a row and shared memory of a tile.
void slice_tile(int op, SliceArgs &a, SliceShape &sh) {
  constexpr size_t kLimit = 227 * 1024 - 256;  // a CTA's shared memory less the static part
  a.rows = slice_rows(op, a.k, a.m, a.n);
  const size_t info = op == RSGPU_OP_RECONSTRUCT ? size_t(a.n) * LaneInfo::kBytes : 0;
  a.wt = 32;
  // 28 threads a row when 256 rows would not fit at 32, and when it lets a
  // second CTA share the SM (128 rows).
  if (size_t(a.rows) * 32 * a.wt + info > kLimit || (a.rows == 128 && !info)) a.wt = 28;
  sh.smem = size_t(a.rows) * 32 * a.wt + info;
}
}  // namespace

uint64_t slice_tile_bytes(int op, uint32_t k, uint32_t m, uint32_t n) {
  SliceArgs a{};
  SliceShape sh;
  a.k = k, a.m = m, a.n = n;
  slice_tile(op, a, sh);
  return 32 * uint64_t(a.wt);
}

int slice_configure(int op, SliceArgs &a, SliceShape &sh) {
  slice_tile(op, a, sh);
  const uint32_t lanes = op == RSGPU_OP_RECONSTRUCT ? a.n : a.m;
  const uint32_t items = std::max(1u, lanes / 4);  // radix-4 groups of a pass: one per warp
  const uint32_t ctas = std::max<uint32_t>(1, uint32_t(227 * 1024 / (sh.smem + 1280)));
  uint32_t warps = 1;
  while (warps * 2 <= items && warps * 2 * ctas <= 32 + 16) warps *= 2;
  sh.threads = int(32 * std::min(warps, 32u));
  const void *fn = reinterpret_cast<const void *>(slice_kernel(op, a.wt));
  RS_CUDA(ensure_smem_limit(fn, sh.smem));
  int per_sm = 0;
  RS_CUDA(blocks_per_sm(fn, sh.threads, sh.smem, &per_sm));
  const uint64_t tile = uint64_t(32) * a.wt;
  const uint64_t tiles = a.items ? a.n_items : ((a.len + tile - 1) / tile) * std::max<uint32_t>(a.n_jobs, 1);
  sh.grid = int(std::min<uint64_t>(tiles, uint64_t(std::max(per_sm, 1)) * device_sm_count()));
  return RSGPU_OK;
}

int slice_launch(int op, const SliceArgs &a, const SliceShape &sh, cudaStream_t s) {
  slice_kernel(op, a.wt)<<<sh.grid, sh.threads, sh.smem, s>>>(a);
  launch_counter_add(1);
  return cuda_status(cudaGetLastError());
}

void slice_elements(int bits, const uint16_t *exp, uint32_t order, uint16_t *out) {
  for (uint32_t i = 0; i < order; ++i)
    out[i] = uint16_t(bits == 8 ? cantor_to_tower<8>(exp[i]) : cantor_to_tower<16>(exp[i]));
}

}  // namespace rsgpu
