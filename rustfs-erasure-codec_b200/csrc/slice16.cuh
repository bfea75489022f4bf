// slice16.cuh -- Leopard GF(2^16) transforms on bit planes.
//
// The arithmetic of slice_fft.cuh on 16 planes (slice_field.cuh), one column
// tile being 32 threads x 32 elements, i.e. 2 KiB of every shard.  A row
// (lane) of a tile is 2 KiB, so all lanes of a wide code do not fit on chip,
// and a transform over 2^b lanes is split in two levels, as a large FFT is:
// 2^bl consecutive lanes (the low layers) and 2^bh lanes 2^bl apart (the high
// layers), each level a tile of rows in shared memory.  Between the levels the
// rows pass through a scratch buffer in plane form, a chunk of tiles at a time
// (how many: leo_slice.hpp).
//
//   encode:  low IFFT of every data group (A) -> V; per residue, high IFFT of
//            every group, their XOR, high FFT (B) -> U; low FFT (C) -> parity
//   decode:  low IFFT of the scaled present shards (A) -> V; per residue, high
//            IFFT, the derivative's high part, high FFT (B) -> U; the
//            derivative's low part, low FFT, scaling (C) -> targets
//
// The formal derivative W + N W, N_t W(l) = W(l | 2^t) over the zero bits t of
// l, splits into high and low bits.  The low part only moves values between
// lanes of one low group and the high FFT acts on every residue alike, so they
// commute, and the high FFT undoes the high IFFT: with W = IFFT_high(V),
//   FFT_high(W + N_high W + N_low W) = FFT_high((1 + N_high) IFFT_high V) + N_low V.
// So B needs no lane of another residue and C adds N_low V to B's result
// (src/core/leopard_gf16/decode.rs:704-910, encode.rs:109-252).
//
// Constants: lane position r + off over distance d as in slice_fft.cuh; below
// 4096 in A and C (three nibbles), below 256 in B: elements of GF(256), so B works
// on the two halves of the planes separately (Sub16).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "apply_tile.cuh"
#include "leo_types.hpp"
#include "slice_fft.cuh"

namespace rsgpu {
namespace {

constexpr uint32_t kRow16 = 2048;  // bytes of a row: 4 quarters of 16 bytes a thread

// x ^= c * y for a constant of three nibbles (two pairs), and of four.
__device__ __forceinline__ void mac16x2(uint32_t c, uint32_t *x0, const uint32_t *y0, uint32_t *x1,
                                        const uint32_t *y1) {
  mac2_nibble<16, 0>(c & 15, x0, y0, x1, y1);
  mac2_nibble<16, 4>((c >> 4) & 15, x0, y0, x1, y1);
  mac2_nibble<16, 8>((c >> 8) & 15, x0, y0, x1, y1);
}
__device__ __forceinline__ void mac16(uint32_t c, uint32_t *x, const uint32_t *y) {
  mac_nibble<16, 0>(c & 15, x, y);
  mac_nibble<16, 4>((c >> 4) & 15, x, y);
  mac_nibble<16, 8>((c >> 8) & 15, x, y);
  mac_nibble<16, 12>(c >> 12, x, y);
}

// Rows in shared memory; base: this thread's words of row 0.
__device__ __forceinline__ void row16_load(uint32_t addr, uint32_t *v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 a = lds_words(addr + q * 512);
    v[4 * q] = a.x, v[4 * q + 1] = a.y, v[4 * q + 2] = a.z, v[4 * q + 3] = a.w;
  }
}
__device__ __forceinline__ void row16_store(uint32_t addr, const uint32_t *v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) sts_words(addr + q * 512, make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
}
// The same in the scratch buffer (p: this thread's words).
__device__ __forceinline__ void row16_get(const uint4 *p, uint32_t *v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 a = p[q * 32];
    v[4 * q] = a.x, v[4 * q + 1] = a.y, v[4 * q + 2] = a.z, v[4 * q + 3] = a.w;
  }
}
__device__ __forceinline__ void row16_put(uint4 *p, const uint32_t *v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) p[q * 32] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}
struct ScratchRows {
  const uint4 *p;
  __device__ __forceinline__ void get(const uint32_t *row, uint32_t (*v)[16]) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) row16_get(p + row[j] * 128, v[j]);
  }
};
__device__ __forceinline__ void copy_row_in(uint32_t addr, const uint4 *p) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(addr + q * 512), "l"(p + q * 32) : "memory");
}
__device__ __forceinline__ void zero_row(uint32_t addr) {
#pragma unroll
  for (int q = 0; q < 4; ++q) sts_words(addr + q * 512, make_uint4(0, 0, 0, 0));
}

// One pass over `rows` rows: two layers (radix 4, distances d = 2^lgd and 2d)
// on rows l, l + d, l + 2d, l + 3d, or with !pair the outer layer alone
// (distance 2^lgd >= 2) on rows l, l + 1 and their partners.  Positions: row i
// stands at off + i; where not null, `in` gives the rows (an IFFT's skipped ones
// are zero) and `out` (this thread's scratch rows) takes them; a group starting
// at or past `limit` rows is skipped, and so is one with no 4-row block in
// `need`.  Both layers go through one copy of the networks (the loop below), with
// the middle rows exchanged in between: two copies, 34 KB each, overflowed the
// instruction cache.
template <bool FWD, class In>
__device__ __forceinline__ void pass16(uint32_t s, const In *in, uint4 *out, uint32_t rows, uint32_t lgd, bool pair,
                                       uint32_t off, uint32_t limit, uint32_t need) {
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t d = 1u << lgd, span = pair ? 4 * d : 2 * d;  // rows of a block
  const uint32_t block = span >= 128 ? ~0u : (1u << (span >> 2)) - 1;
#pragma unroll 1
  for (uint32_t q = warp; q < (rows >> 2); q += warps) {
    // Rows in load order, a layer pairing row[0] with row[1] and row[2] with
    // row[3]: the inner layer's pairs for an IFFT, the outer layer's for an FFT.
    uint32_t r, row[4];
    if (pair) {
      r = (q >> lgd) << (lgd + 2);
      const uint32_t l = r + (q & (d - 1));
      row[0] = l, row[1] = FWD ? l + 2 * d : l + d, row[2] = FWD ? l + d : l + 2 * d, row[3] = l + 3 * d;
    } else {
      r = (q >> (lgd - 1)) << (lgd + 1);
      const uint32_t l = r + 2 * (q & (d / 2 - 1));
      row[0] = l, row[1] = l + d, row[2] = l + 1, row[3] = l + d + 1;
    }
    if (r >= limit || !((need >> (r >> 2)) & block)) {  // warp-uniform
      if (!FWD && in)
        for (int j = 0; j < 4; ++j) zero_row(s + row[j] * kRow16);
      continue;
    }
    const uint32_t e_in = tower_const<16>((r + off) >> lgd), e_out = pair ? tower_const<16>((r + off) >> (lgd + 1)) : e_in;
    uint32_t v[4][16];
    if (in) {  // CTA-uniform
      in->get(row, v);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) row16_load(s + row[j] * kRow16, v[j]);
    }
#pragma unroll 1
    for (int step = pair ? 0 : 1; step < 2; ++step) {
      const bool inner = FWD ? pair && step == 1 : step == 0;
      if (!FWD) {
        xor_planes<16>(v[1], v[0]);
        xor_planes<16>(v[3], v[2]);
      }
      mac16x2(inner ? e_in : e_out, v[0], v[1], v[2], v[3]);
      if (inner) mac_const<16, 2>(v[2], v[3]);
      if (FWD) {
        xor_planes<16>(v[1], v[0]);
        xor_planes<16>(v[3], v[2]);
      }
      if (step == 0) {  // the other layer pairs the rows crosswise
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t t = v[1][i];
          v[1][i] = v[2][i];
          v[2][i] = t;
        }
        const uint32_t t = row[1];
        row[1] = row[2];
        row[2] = t;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (out)  // CTA-uniform
        row16_put(out + row[j] * 128, v[j]);
      else
        row16_store(s + row[j] * kRow16, v[j]);
    }
  }
}
// IFFT over 2^b rows (b >= 3); the first pass reads `in`, unless null, the
// last one writes out, shared memory is in between.
template <class In>
__device__ __forceinline__ void ifft16(uint32_t rows, const In *in, uint4 *out, uint32_t b, uint32_t off,
                                       uint32_t limit) {
#pragma unroll 1
  for (uint32_t lgd = 0; lgd < b; lgd += 2) {
    const bool last = lgd + 2 >= b;
    pass16<false>(rows, lgd ? nullptr : in, last ? out : nullptr, 1u << b, lgd, lgd + 1 < b, off,
                      last ? ~0u : limit, ~0u);
    __syncthreads();
  }
}
// FFT over 2^b rows into shared memory; the first pass reads `in`, unless null.
__device__ __forceinline__ void fft16(uint32_t rows, const ScratchRows *in, uint32_t b, uint32_t off, uint32_t limit,
                                      uint32_t need) {
  const uint32_t odd = b & 1;
#pragma unroll 1
  for (int lgd = int(b) - 2 + int(odd); lgd >= 0; lgd -= 2) {
    const bool single = odd && lgd == int(b) - 1;
    pass16<true>(rows, in, nullptr, 1u << b, uint32_t(lgd), !single, off, single ? ~0u : limit, single ? ~0u : need);
    in = nullptr;
    __syncthreads();
  }
}

// The derivative's low part over the n >= 4 rows of `in` (this thread's scratch
// rows): N V + add, into shared memory.  A warp takes 4 consecutive rows; `add`
// is on its way while the rows it needs of the other warps are copied.  A CTA
// has a warp for every 4 rows.
__device__ __forceinline__ void derivative16(uint32_t rows, uint32_t n, const uint4 *in, const uint4 *add) {
  const uint32_t warp = threadIdx.x >> 5, items = n >> 2;
  const uint32_t R = min(warp, items - 1) << 2;  // past the last: redone, not stored
  const uint32_t base = rows + R * kRow16;
  if (warp < items) {
#pragma unroll
    for (int j = 0; j < 4; ++j) copy_row_in(base + j * kRow16, in + (R + j) * 128);
  }
  uint32_t v[4][16], u[16];
#pragma unroll
  for (int j = 0; j < 4; ++j) row16_get(add + (R + j) * 128, v[j]);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  row16_load(base + kRow16, u);
  xor_planes<16>(v[0], u);
  row16_load(base + 2 * kRow16, u);
  xor_planes<16>(v[0], u);
  row16_load(base + 3 * kRow16, u);
  xor_planes<16>(v[1], u);
  xor_planes<16>(v[2], u);
#pragma unroll 1
  for (uint32_t t = 4; t < n; t <<= 1) {
    if (R & t) continue;  // warp-uniform
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      row16_load(base + (t + j) * kRow16, u);
      xor_planes<16>(v[j], u);
    }
  }
  __syncthreads();
  if (warp < items) {
#pragma unroll
    for (int j = 0; j < 4; ++j) row16_store(base + j * kRow16, v[j]);
  }
  __syncthreads();
}

// A thread's 32 elements of a tile: low and high bytes of half h of blocks
// t / 2 and 16 + t / 2 (h = t & 1), so two threads read 32 contiguous bytes.
// A 64-byte block holds the low bytes of its 32 elements, then the high ones.
struct Cols16 {
  uint64_t a, b;
  bool on_a, on_b;
  __device__ __forceinline__ Cols16(uint64_t tile, uint32_t t, uint64_t len) {
    a = tile + 64ull * (t >> 1) + 16 * (t & 1);
    b = a + 1024;
    on_a = a < len;
    on_b = b < len;
  }
  __device__ __forceinline__ void load(const uint8_t *p, uint32_t *v) const {
    uint4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = make_uint4(0, 0, 0, 0);
    if (p && on_a) x[0] = ld_stream(p + a), x[2] = ld_stream(p + a + 32);
    if (p && on_b) x[1] = ld_stream(p + b), x[3] = ld_stream(p + b + 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[4 * i] = x[i].x, v[4 * i + 1] = x[i].y, v[4 * i + 2] = x[i].z, v[4 * i + 3] = x[i].w;
  }
  __device__ __forceinline__ static void planes(uint32_t *v) {
    slice8(v);
    slice8(v + 8);
    planes_to_tower<16>(v);
  }
  // Planes to bytes: x holds the chunks in load's order.
  __device__ __forceinline__ static void bytes(uint32_t *v) {
    planes_to_cantor<16>(v);
    slice8(v);
    slice8(v + 8);
  }
  __device__ __forceinline__ void store(uint8_t *p, const uint32_t *v) const {
    auto w = [&](int i) { return make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]); };
    if (on_a) st_stream(p + a, w(0)), st_stream(p + a + 32, w(2));
    if (on_b) st_stream(p + b, w(1)), st_stream(p + b + 32, w(3));
  }
  __device__ __forceinline__ uint32_t compare(const uint8_t *p, const uint32_t *v) const {
    uint32_t bad = 0;
    auto diff = [&](const uint8_t *s, int i) {
      const uint4 u = ld_stream(s);
      bad |= (u.x ^ v[4 * i]) | (u.y ^ v[4 * i + 1]) | (u.z ^ v[4 * i + 2]) | (u.w ^ v[4 * i + 3]);
    };
    if (on_a) diff(p + a, 0), diff(p + a + 32, 2);
    if (on_b) diff(p + b, 1), diff(p + b + 32, 3);
    return bad;
  }
};

}  // namespace
}  // namespace rsgpu
