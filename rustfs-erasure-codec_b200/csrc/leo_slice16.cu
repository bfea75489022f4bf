// leo_slice16.cu -- launches of the bit-sliced Leopard GF(2^16) transforms
// (slice16.cuh).
#include <cuda_runtime.h>

#include <algorithm>

#include "codec.hpp"
#include "launch_cfg.hpp"
#include "leo_slice.hpp"
#include "slice16.cuh"

namespace rsgpu {

#define RS_CUDA(expr)                              \
  do {                                             \
    cudaError_t e_ = (expr);                       \
    if (e_ != cudaSuccess) return cuda_status(e_); \
  } while (0)

namespace {


// A work item of a launch: group `grp` of tile `x` of the chunk.
struct Item16 {
  uint32_t grp, x, job;
  uint64_t col;
};
__device__ __forceinline__ Item16 item16(const Slice16Args &a, uint32_t it, uint32_t groups) {
  Item16 w;
  w.x = it / groups;
  w.grp = it - w.x * groups;
  const uint32_t tile = a.tile0 + w.x;
  w.job = tile / a.tiles_per_job;
  w.col = uint64_t(tile - w.job * a.tiles_per_job) * kRow16;
  return w;
}

// What a warp needs of 32 consecutive lanes, lane l0 + t in thread t: all
// looked up at once, then handed out by shuffles.
struct Lanes16 {
  uint64_t ptr;  // shard (0: nothing to do)
  uint32_t c;    // tower constant of its scaling
  // ROLE: 0 encode input, 1 decode input, 2 decode target, 3 parity output.
  template <int ROLE>
  __device__ __forceinline__ static Lanes16 get(const Slice16Args &a, const LeoJob &jd, uint32_t l) {
    Lanes16 w{0, 0};
    int sh = -1;
    if (ROLE == 0) {
      if (l < a.k) sh = int(l);
    } else if (ROLE == 3) {
      if (l < a.p) sh = int(a.k + l);
    } else {
      sh = l < a.p ? int(a.k + l) : l >= a.m && l < a.m + a.k ? int(l - a.m) : -1;
      if (sh >= 0 && jd.role[sh] != ROLE) sh = -1;
    }
    if (sh >= 0) {
      w.ptr = reinterpret_cast<uint64_t>(a.ptrs[jd.ptr_off + sh]);
      if (ROLE == 1) w.c = a.elem[jd.err[l]];
      if (ROLE == 2) w.c = a.elem[a.mod - jd.err[l]];
    }
    return w;
  }
  __device__ __forceinline__ Lanes16 at(uint32_t i) const {
    return Lanes16{__shfl_sync(0xffffffffu, ptr, int(i)), __shfl_sync(0xffffffffu, c, int(i))};
  }
};

// An encode's data lanes straight into the first pass, four in flight at once
// (75 -> 72 us a chunk of 64 tiles of 1024+512).  A decode goes through shared
// memory, lane by lane: the scaling and the absent third of the lanes cost more
// in the pass (88 us a chunk; 102 in the pass, more with absent lanes skipped).
struct DataRows {
  const Slice16Args &a;
  const LeoJob &jd;
  uint32_t R;
  Cols16 cols;
  __device__ __forceinline__ void get(const uint32_t *row, uint32_t (*v)[16]) const {
    const Lanes16 lanes = Lanes16::get<0>(a, jd, R + row[0] + (threadIdx.x & 3));
#pragma unroll
    for (int j = 0; j < 4; ++j) cols.load(reinterpret_cast<const uint8_t *>(lanes.at(j).ptr), v[j]);
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      Cols16::planes(v[0]);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t x = v[0][i];
        v[0][i] = v[1][i];
        v[1][i] = v[2][i];
        v[2][i] = v[3][i];
        v[3][i] = x;
      }
    }
  }
};

// A: low IFFT of 2^bl consecutive lanes, shards -> V.  Decode: lane l is
// parity l or data l - m, scaled by its locator.  Encode: lane l is data l,
// at position m + l.
template <bool DEC>
__global__ void __launch_bounds__(512, 1) k_slice16_a(Slice16Args a) {
  extern __shared__ __align__(16) uint4 smem16[];
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, t = threadIdx.x & 31;
  const uint32_t rows = 1u << a.bl;
  const uint32_t sbase = uint32_t(__cvta_generic_to_shared(smem16)) + 16 * t;
  const uint32_t groups = a.v_rows >> a.bl;
#pragma unroll 1
  for (uint32_t it = blockIdx.x; it < a.tiles * groups; it += gridDim.x) {
    const Item16 w = item16(a, it, groups);
    const LeoJob jd = a.jobs[w.job];
    const uint32_t R = w.grp << a.bl, limit = DEC ? jd.input_count : a.k;
    if (R >= limit) continue;  // CTA-uniform: zero lanes, never read
    const Cols16 cols(w.col, t, a.len);
    if (DEC) {
#pragma unroll 1
      for (uint32_t i0 = 0; i0 < rows; i0 += 32) {
        const Lanes16 lanes = Lanes16::get<1>(a, jd, R + i0 + t);
#pragma unroll 1
        for (uint32_t i = warp; i < min(rows - i0, 32u); i += warps) {
          const Lanes16 lane = lanes.at(i);
          uint32_t x[16] = {};
          if (lane.ptr) {  // warp-uniform
            uint32_t y[16];
            cols.load(reinterpret_cast<const uint8_t *>(lane.ptr), y);
            Cols16::planes(y);
            mac16(lane.c, x, y);
          }
          row16_store(sbase + (i0 + i) * kRow16, x);
        }
      }
      __syncthreads();
    }
    const DataRows in{a, jd, R, cols};
    ifft16(sbase, DEC ? nullptr : &in, a.v + (size_t(w.x) * a.v_rows + R) * 128 + t, a.bl, DEC ? R : a.m + R,
              limit - R);
  }
}

// Half rows in the scratch buffer, `step` uint4 apart: what the first pass of B
// reads and the last one writes.
struct ScratchIn {
  const uint4 *p;
  size_t step;
  uint32_t live;  // rows past it are zero
  __device__ __forceinline__ void get(uint32_t r, uint32_t j, uint32_t *v) const {
    uint4 x = make_uint4(0, 0, 0, 0), y = x;
    if (r + j < live) x = p[(r + j) * step], y = p[(r + j) * step + 32];  // warp-uniform
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
  }
};
struct FirstRows : Rows<32> {  // a skipped group's rows are zero
  __device__ __forceinline__ FirstRows(const Rows<32> &r) : Rows<32>(r) {}
  __device__ __forceinline__ void skip(uint32_t l, uint32_t d) const {
    const uint32_t zero[8] = {};
    for (uint32_t j = 0; j < 4; ++j) put(l, j * d, zero);
  }
};
struct ScratchOut {
  uint4 *p;
  size_t step;
  uint32_t rows;  // rows past it are not wanted
  __device__ __forceinline__ void put(uint32_t r, uint32_t j, const uint32_t *v) const {
    if (r + j >= rows) return;  // warp-uniform
    p[(r + j) * step] = make_uint4(v[0], v[1], v[2], v[3]);
    p[(r + j) * step + 32] = make_uint4(v[4], v[5], v[6], v[7]);
  }
  __device__ __forceinline__ void skip(uint32_t, uint32_t) const {}
};

// B: the high layers of residue c (lanes c + 2^bl * j), V -> U.  All constants
// lie in GF(256), which maps the low and the high 8 planes to themselves, so
// the two halves of a row are independent 8-plane transforms: half the shared
// memory and registers of 16-plane rows, twice the warps (1024+512, 16 KiB x 16:
// encode 535 -> 476 us, rebuild 1279 -> 1110).  The first pass reads the scratch
// buffer and the last one writes it (64 rows: 83 -> 71 us a chunk of 64 tiles).
template <bool DEC>
__global__ void __launch_bounds__(512, 2) k_slice16_b(Slice16Args a) {
  extern __shared__ __align__(16) uint4 smem16[];
  const uint32_t t = threadIdx.x & 31;
  const uint32_t rows = 1u << a.bh, residues = 1u << a.bl, b = a.bh, odd = b & 1;
  const uint32_t sbase = uint32_t(__cvta_generic_to_shared(smem16));
  const Rows<32> acc(sbase, t), tmp(sbase + rows * Rows<32>::kStride, t);
  const size_t step = size_t(residues) * 128;  // one j on
#pragma unroll 1
  for (uint32_t it = blockIdx.x; it < a.tiles * residues * 2; it += gridDim.x) {
    const Item16 w = item16(a, it >> 1, residues);
    const uint32_t half = (it & 1) * 64 + t;
    const uint4 *vin = a.v + (size_t(w.x) * a.v_rows + w.grp) * 128 + half;
    const ScratchOut uout{a.u + (size_t(w.x) * a.u_rows + w.grp) * 128 + half, step, a.u_rows >> a.bl};
    uint32_t lgd = 2;  // layers done by the IFFT, then left to the FFT
    if (DEC) {
      const uint32_t live = (a.jobs[w.job].input_count + residues - 1) >> a.bl;  // groups A wrote
      // Layers 0 .. b - 3 (an odd b: layer 2 alone), the middle, and back.
      slice_pass4<32, false, Sub16>(ScratchIn{vin, step, live}, FirstRows(acc), false, rows, 0, 0, live, ~0ull);
      __syncthreads();
      if (odd) {
        slice_pass2<32, false, Sub16>(acc, acc, false, rows, lgd++, 0);
        __syncthreads();
      }
#pragma unroll 1
      for (; lgd < b - 2; lgd += 2) {
        slice_pass4<32, false, Sub16>(acc, acc, false, rows, lgd, 0, live, ~0ull);
        __syncthreads();
      }
      slice_middle<32, Sub16>(acc, rows);
    } else {
      const uint32_t groups = (a.k + a.m - 1) / a.m;
#pragma unroll 1
      for (uint32_t g = 0; g < groups; ++g) {
        const uint32_t live = min(rows, ((a.k - g * a.m) + residues - 1) >> a.bl), off = rows * (1 + g);
        const Rows<32> &dst = g ? tmp : acc;
        slice_pass4<32, false, Sub16>(ScratchIn{vin + size_t(g) * rows * step, step, live}, FirstRows(dst), false, rows,
                                      0, off, live, ~0ull);
        __syncthreads();
#pragma unroll 1
        for (lgd = 2; lgd + 2 <= b; lgd += 2) {
          const bool last = lgd + 2 == b;
          slice_pass4<32, false, Sub16>(dst, last ? acc : dst, last && g, rows, lgd, off, last ? ~0u : live, ~0ull);
          __syncthreads();
        }
        if (odd) {
          slice_pass2<32, false, Sub16>(dst, acc, g != 0, rows, lgd, off);
          __syncthreads();
        }
      }
      if (odd) {
        slice_pass2<32, true, Sub16>(acc, acc, false, rows, b - 1, 0);
        __syncthreads();
      }
      lgd = b - odd;
    }
#pragma unroll 1
    for (; lgd > 2 + (DEC ? odd : 0u); lgd -= 2) {
      slice_pass4<32, true, Sub16>(acc, acc, false, rows, lgd - 2, 0, uout.rows, ~0ull);
      __syncthreads();
    }
    if (DEC && odd) {
      slice_pass2<32, true, Sub16>(acc, acc, false, rows, 2, 0);
      __syncthreads();
    }
    slice_pass4<32, true, Sub16>(acc, uout, false, rows, 0, 0, uout.rows, ~0ull);
    __syncthreads();
  }
}

// C: low FFT of 2^bl consecutive lanes, U (decode: plus N_low V) -> outputs.
// MODE: 0 encode, 1 verify, 2 decode.
template <int MODE>
__global__ void __launch_bounds__(512, 1) k_slice16_c(Slice16Args a) {
  extern __shared__ __align__(16) uint4 smem16[];
  __shared__ uint32_t s_need;
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, t = threadIdx.x & 31;
  const uint32_t rows = 1u << a.bl;
  const uint32_t sbase = uint32_t(__cvta_generic_to_shared(smem16)) + 16 * t;
  const uint32_t groups = a.u_rows >> a.bl;
#pragma unroll 1
  for (uint32_t it = blockIdx.x; it < a.tiles * groups; it += gridDim.x) {
    const Item16 w = item16(a, it, groups);
    const LeoJob jd = a.jobs[w.job];
    const uint32_t R = w.grp << a.bl;
    uint32_t need = ~0u;
    if (MODE == 2) {
      // 4-lane blocks of the group that hold a target.
      if (threadIdx.x < 32) {
        uint32_t bits = 0;
        for (uint32_t i = t; i < rows; i += 32) {
          const uint32_t l = R + i;
          const int sh = l < a.p ? int(a.k + l) : l >= a.m && l < a.m + a.k ? int(l - a.m) : -1;
          if (sh >= 0 && jd.role[sh] == 2) bits |= 1u << (i >> 2);
        }
        bits = __reduce_or_sync(0xffffffffu, bits);
        if (t == 0) s_need = bits;
      }
      __syncthreads();
      need = s_need;
      if (!need) {  // CTA-uniform
        __syncthreads();  // s_need is read before the next item writes it
        continue;
      }
    }
    const ScratchRows uin{a.u + (size_t(w.x) * a.u_rows + R) * 128 + t};
    const bool derive = MODE == 2 && R < jd.input_count;  // CTA-uniform; past it V is zero
    if (derive) derivative16(sbase, rows, a.v + (size_t(w.x) * a.v_rows + R) * 128 + t, uin.p);
    fft16(sbase, derive ? nullptr : &uin, a.bl, R, (MODE == 2 ? a.m + a.k : a.p) - R, need);
    const Cols16 cols(w.col, t, a.len);
    uint32_t bad = 0;
#pragma unroll 1
    for (uint32_t i0 = 0; i0 < rows; i0 += 32) {
      const Lanes16 lanes = Lanes16::get<MODE == 2 ? 2 : 3>(a, jd, R + i0 + t);
#pragma unroll 1
      for (uint32_t i = warp; i < min(rows - i0, 32u); i += warps) {
        const Lanes16 lane = lanes.at(i);
        if (!lane.ptr) continue;  // warp-uniform
        uint8_t *out = reinterpret_cast<uint8_t *>(lane.ptr);
        uint32_t v[16];
        row16_load(sbase + (i0 + i) * kRow16, v);
        if (MODE == 2) {
          uint32_t x[16] = {};
          mac16(lane.c, x, v);
          Cols16::bytes(x);
          cols.store(out, x);
        } else {
          Cols16::bytes(v);
          if (MODE == 1)
            bad |= cols.compare(out, v);
          else
            cols.store(out, v);
        }
      }
    }
    if (MODE == 1 && __any_sync(0xffffffffu, bad) && t == 0) atomicOr(a.flags + jd.flag_idx, 1u);
    __syncthreads();
  }
}

using Kernel16 = void (*)(Slice16Args);
struct Launch16 {
  Kernel16 fn;
  int threads;
  size_t smem;
  uint32_t groups;  // work items a tile
};
// One warp for every radix-4 group.  A and C hold 128 registers a thread, so 16
// warps an SM, in CTAs of 1 (4 rows) to 16 warps (64 rows).  With CTAs of 8 warps
// for 16 rows, half of them idle in the passes, 1024+512 encode of 16 KiB x 16
// took 476 us; with 4 warps and direct scratch access 370.
void launches16(int op, const Slice16Args &a, Launch16 *out) {
  const bool dec = op == RSGPU_OP_RECONSTRUCT;
  const int low = 32 << a.bl >> 2, high = 32 << a.bh >> 2;
  const size_t smem = size_t(kRow16) << a.bl, half = size_t(kRow16 / 2) << a.bh;
  out[0] = Launch16{dec ? k_slice16_a<true> : k_slice16_a<false>, low, smem, a.v_rows >> a.bl};
  out[1] = Launch16{dec ? k_slice16_b<true> : k_slice16_b<false>, high, dec || a.k <= a.m ? half : 2 * half, 2u << a.bl};
  out[2] = Launch16{dec ? k_slice16_c<2> : op == RSGPU_OP_VERIFY ? k_slice16_c<1> : k_slice16_c<0>, low, smem,
                    a.u_rows >> a.bl};
}

uint32_t log2u(uint32_t v) {
  uint32_t b = 0;
  while ((2u << b) <= v) ++b;
  return b;
}

}  // namespace

bool slice16_configure(int op, Slice16Args &a) {
  const bool dec = op == RSGPU_OP_RECONSTRUCT;
  const uint32_t b = log2u(dec ? a.n : a.m);
  if (!slice16_pays(op, a.k, a.m, a.n, a.len, a.n_jobs)) return false;
  a.bl = dec ? std::min(b / 2, b - 4) : std::max(b / 2, b - 5);
  a.bh = b - a.bl;
  if (a.bl > 6 || a.bh > 6) return false;
  const uint32_t low = 1u << a.bl;
  auto up = [&](uint32_t v) { return (v + low - 1) & ~(low - 1); };
  a.v_rows = dec ? up(a.m + a.k) : up(a.k);
  a.u_rows = dec ? up(a.m + a.k) : up(a.p);
  // Positions of the constants (slice16.cuh).
  const uint32_t top = dec ? a.n : a.m + (a.k + a.m - 1) / a.m * a.m;
  if (top > 4096 || (top >> a.bl) > 256) return false;
  a.tiles_per_job = uint32_t((a.len + kRow16 - 1) / kRow16);
  return true;
}

static size_t tile_bytes16(const Slice16Args &a) { return (size_t(a.v_rows) + a.u_rows) * kRow16; }
static uint64_t most_tiles16(const Slice16Args &a) { return std::max<uint64_t>(a.max_scratch / tile_bytes16(a), 1); }

size_t slice16_scratch_limit(const Slice16Args &a) { return most_tiles16(a) * tile_bytes16(a); }

size_t slice16_scratch_bytes(const Slice16Args &a, uint64_t tiles) {
  const uint64_t chunks = (tiles + most_tiles16(a) - 1) / most_tiles16(a);
  return size_t(chunks ? (tiles + chunks - 1) / chunks : 1) * tile_bytes16(a);
}

namespace {
// Tiles of a chunk.
uint32_t chunk16(const Slice16Args &a) {
  return uint32_t(slice16_scratch_bytes(a, uint64_t(a.tiles_per_job) * a.n_jobs) / tile_bytes16(a));
}
}  // namespace

uint64_t slice16_kernels(const Slice16Args &a) {
  const uint32_t chunk = chunk16(a);
  return 3 * ((uint64_t(a.tiles_per_job) * a.n_jobs + chunk - 1) / chunk);
}

int slice16_launch(int op, Slice16Args a, void *scratch, cudaStream_t s) {
  Launch16 step[3];
  launches16(op, a, step);
  const uint64_t total = uint64_t(a.tiles_per_job) * a.n_jobs;
  const uint32_t chunk = chunk16(a);
  a.v = static_cast<uint4 *>(scratch);
  a.u = a.v + size_t(chunk) * a.v_rows * (kRow16 / 16);
  uint64_t launched = 0;
  for (uint64_t t0 = 0; t0 < total; t0 += chunk) {
    a.tile0 = uint32_t(t0);
    a.tiles = uint32_t(std::min<uint64_t>(chunk, total - t0));
    for (const Launch16 &l : step) {
      const void *fn = reinterpret_cast<const void *>(l.fn);
      RS_CUDA(ensure_smem_limit(fn, l.smem));
      int per_sm = 0;
      RS_CUDA(blocks_per_sm(fn, l.threads, l.smem, &per_sm));
      const uint64_t items = uint64_t(a.tiles) * l.groups;
      const int grid = int(std::min<uint64_t>(items, uint64_t(std::max(per_sm, 1)) * device_sm_count()));
      l.fn<<<grid, l.threads, l.smem, s>>>(a);
      ++launched;
    }
  }
  launch_counter_add(launched);
  return cuda_status(cudaGetLastError());
}

}  // namespace rsgpu
