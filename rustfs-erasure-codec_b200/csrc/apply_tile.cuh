// apply_tile.cuh -- device code of the classic matrix-apply kernel (K1), one
// column tile at a time, shared by k_apply_vec (k_classic.cu) and the
// mixed-batch persistent kernel (batch.cu).
//
// out[r] = sum_j c[r][j] * in[j] over GF(2^8), bytewise.  Each thread owns 16
// (or 32) byte columns of one stripe and reads every input shard exactly once
// with coalesced 128-bit loads.  Products are table lookups split over the
// bits of the data byte, and the tables of four outputs are packed into one
// 32-bit word per entry, so one lookup serves four output rows.  A lookup is a
// warp shuffle into a 32-entry table held one entry per lane; how bytes share
// lookups is described at Lut below.  The staged tile of k_classic.cu uses
// pairs of 16-entry tables instead (4+4 split; a table mirrored into lanes
// 16..31 makes the raw shifted data word a valid index).
// All outputs of a column are accumulated in registers and written once.
// The tables need not come from the classic field: any GF(2)-linear byte map
// (multiplication by a constant in the Leopard GF(2^8) field, for one) packs
// the same way.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.hpp"

namespace rsgpu {
namespace {

__device__ __forceinline__ uint32_t tshfl(uint32_t table, uint32_t idx) {
  uint32_t r;
  asm("shfl.sync.idx.b32 %0, %1, %2, 31, -1;" : "=r"(r) : "r"(table), "r"(idx));
  return r;
}

// Accumulate the four columns of data word w into a[0..3] (four packed outputs each).
__device__ __forceinline__ void mac4(uint32_t w, uint32_t lo, uint32_t hi, uint32_t *a) {
  a[0] ^= tshfl(lo, w) ^ tshfl(hi, w >> 4);
  a[1] ^= tshfl(lo, w >> 8) ^ tshfl(hi, w >> 12);
  a[2] ^= tshfl(lo, w >> 16) ^ tshfl(hi, w >> 20);
  a[3] ^= tshfl(lo, w >> 24) ^ tshfl(hi, w >> 28);
}

// Transpose 4 columns x 4 packed outputs into 4 output words.
__device__ __forceinline__ void transpose4(const uint32_t *a, uint32_t *o) {
  uint32_t t0 = __byte_perm(a[0], a[1], 0x5140);
  uint32_t t1 = __byte_perm(a[2], a[3], 0x5140);
  uint32_t t2 = __byte_perm(a[0], a[1], 0x7362);
  uint32_t t3 = __byte_perm(a[2], a[3], 0x7362);
  o[0] = __byte_perm(t0, t1, 0x5410);
  o[1] = __byte_perm(t0, t1, 0x7632);
  o[2] = __byte_perm(t2, t3, 0x5410);
  o[3] = __byte_perm(t2, t3, 0x7632);
}

// 5+3 split, PRMT half: selector nibble c = high three bits of byte c of w.
// y = x | (x >> 4) puts byte i + 1's field in the high nibble of byte i; the
// fields do not overlap, so it equals x + (x >> 4), which one multiply-high
// and add computes on the FMA pipe (the GF(2^8) transforms are bound by the
// integer pipe).
__device__ __forceinline__ uint32_t hi3_selector(uint32_t w) {
  const uint32_t x = (w >> 5) & 0x07070707u;
  const uint32_t y = __umulhi(x, 1u << 28) + x;
  return __byte_perm(y, 0, 0x3320);
}

__device__ __forceinline__ uint4 ld_stream(const uint8_t *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ void st_stream(uint8_t *p, uint4 v) {
  asm volatile("st.global.L1::no_allocate.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

// ------------------------------------------------------------------ shared lookups
// Lookup tables of C inputs (C = 1, 3 or 5) for four packed outputs, one entry
// of 32 per lane.  A shuffle reads a table of 32 entries, i.e. five bits of
// data, so looking bytes up one by one (two lookups each) wastes two bits of
// ten.  Here each byte's low five bits index its input's own table and the
// high bits of several inputs, three each, are packed five to a lookup: five
// inputs take 5 + 3 lookups a column instead of 10, three take 3 + 2.  The
// packing is done on whole words (four columns at once), so the integer work
// per lookup stays where it was.
//   mixed index 0: bits 5-7 of input 0, bits 5-6 of input 1
//   mixed index 1: bit 7 of input 1, bits 5-7 of input 2, bit 5 of input 3
//   mixed index 2: bits 6-7 of input 3, bits 5-7 of input 4
template <int C>
struct Lut {
  static constexpr int kMixed = (3 * C + 4) / 5;
  uint32_t low[C], mix[kMixed];
};

// tab(i, w): word w of input i's packed table (layout of common.hpp; words
// 16..63 are used: 16 + n holds c * (n << 4), 32 + n holds c * n).
template <int C, class T>
__device__ __forceinline__ void lut_load(Lut<C> &t, uint32_t lane, T tab) {
#pragma unroll
  for (int i = 0; i < C; ++i) t.low[i] = tab(i, 32 + lane);
  const uint32_t l = lane;
  if (C == 1) {
    t.mix[0] = tab(0, 16 + 2 * (l & 7));  // repeated: the index's bits 3-4 do not matter
    return;
  }
  t.mix[0] = tab(0, 16 + 2 * (l & 7)) ^ tab(1 % C, 16 + 2 * (l >> 3));
  t.mix[1 % Lut<C>::kMixed] = tab(1 % C, 16 + 8 * (l & 1)) ^ tab(2 % C, 16 + 2 * ((l >> 1) & 7));
  if (C == 5) {
    t.mix[1 % Lut<C>::kMixed] ^= tab(3 % C, 16 + 2 * (l >> 4));
    t.mix[2 % Lut<C>::kMixed] = tab(3 % C, 16 + 4 * (l & 3)) ^ tab(4 % C, 16 + 2 * (l >> 2));
  }
}

// Mixed index words of one word of each input.
template <int C>
__device__ __forceinline__ void lut_index(const uint32_t *x, uint32_t *m) {
  if (C == 1) {
    m[0] = x[0] >> 5;
    return;
  }
  m[0] = ((x[0] >> 5) & 0x07070707u) | ((x[1 % C] >> 2) & 0x18181818u);
  uint32_t m1 = ((x[1 % C] >> 7) & 0x01010101u) | ((x[2 % C] >> 4) & 0x0E0E0E0Eu);
  if (C == 5) {
    m1 |= (x[3 % C] >> 1) & 0x10101010u;
    m[2 % Lut<C>::kMixed] = ((x[3 % C] >> 6) & 0x03030303u) | ((x[4 % C] >> 3) & 0x1C1C1C1Cu);
  }
  m[1 % Lut<C>::kMixed] = m1;
}

// acc[0..3] ^= the products of one word (four columns) of each input.
template <int C>
__device__ __forceinline__ void lut_mac(const Lut<C> &t, const uint32_t *x, const uint32_t *m, uint32_t *acc) {
#pragma unroll
  for (int b = 0; b < 4; ++b) {
#pragma unroll
    for (int i = 0; i < C; ++i) acc[b] ^= tshfl(t.low[i], x[i] >> (8 * b));
#pragma unroll
    for (int i = 0; i < Lut<C>::kMixed; ++i) acc[b] ^= tshfl(t.mix[i], m[i] >> (8 * b));
  }
}

// The lookups of K inputs: fives, then a three, then singles.
template <int K>
struct LutSet {
  static constexpr int kFive = K / 5, kThree = K % 5 >= 3 ? 1 : 0, kOne = K % 5 - 3 * kThree;
  Lut<5> five[kFive ? kFive : 1];
  Lut<3> three;
  Lut<1> one[kOne ? kOne : 1];
  // tbl: the packed table of four outputs over K inputs.
  __device__ __forceinline__ void load(const uint32_t *tbl, uint32_t lane) {
    auto at = [&](int j0) {
      return [=](int i, uint32_t w) { return __ldg(tbl + (j0 + i) * kTableWords + w); };
    };
#pragma unroll
    for (int q = 0; q < kFive; ++q) lut_load<5>(five[q], lane, at(5 * q));
    if (kThree) lut_load<3>(three, lane, at(5 * kFive));
#pragma unroll
    for (int q = 0; q < kOne; ++q) lut_load<1>(one[q], lane, at(5 * kFive + 3 * kThree + q));
  }
  // acc[0..3] ^= the products of one word of every input.
  __device__ __forceinline__ void mac(const uint32_t *x, uint32_t *acc) const {
    uint32_t m[3];
#pragma unroll
    for (int q = 0; q < kFive; ++q) {
      lut_index<5>(x + 5 * q, m);
      lut_mac<5>(five[q], x + 5 * q, m, acc);
    }
    if (kThree) {
      lut_index<3>(x + 5 * kFive, m);
      lut_mac<3>(three, x + 5 * kFive, m, acc);
    }
#pragma unroll
    for (int q = 0; q < kOne; ++q) {
      lut_index<1>(x + 5 * kFive + 3 * kThree + q, m);
      lut_mac<1>(one[q], x + 5 * kFive + 3 * kThree + q, m, acc);
    }
  }
};

// Products of C inputs (x: their loaded words) from j0 on.
template <int C, int NG, int V>
__device__ __forceinline__ void apply_products(const JobDesc &d, uint32_t g0, uint32_t groups, uint32_t j0,
                                               const uint4 (*x)[V], uint32_t lane, uint32_t (*acc)[V][16]);

// Inputs j0 .. j0 + C + D of one tile and pass: loads, tables and products.
// D = 1: one input more that shares no lookups, for what is left of 2 or 4
// inputs.  Its load is on its way with the others; in a step of its own it made
// a thread wait for memory once more (k_mix, 4+2 encode of 256 KiB x 64
// 36.5 -> 33.0 us).
template <int C, int NG, int V, int D = 0>
__device__ __forceinline__ void apply_step(const uint8_t *const *ptr, const JobDesc &d, uint32_t g0, uint32_t groups,
                                           uint32_t j0, const uint64_t *col, const bool *active, uint32_t lane,
                                           uint32_t (*acc)[V][16]) {
  uint4 x[C + D][V];
#pragma unroll
  for (int i = 0; i < C + D; ++i) {
    const uint8_t *src = ptr[j0 + i];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      x[i][v] = make_uint4(0, 0, 0, 0);
      if (active[v]) x[i][v] = ld_stream(src + col[v]);
    }
  }
  apply_products<C, NG, V>(d, g0, groups, j0, x, lane, acc);
  if (D) apply_products<1, NG, V>(d, g0, groups, j0 + C, x + C, lane, acc);
}

template <int C, int NG, int V>
__device__ __forceinline__ void apply_products(const JobDesc &d, uint32_t g0, uint32_t groups, uint32_t j0,
                                               const uint4 (*x)[V], uint32_t lane, uint32_t (*acc)[V][16]) {
  Lut<C> lut[NG];
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const uint32_t *tbl = d.tbl + (size_t(g0 + (uint32_t(g) < groups ? g : 0)) * d.n_in + j0) * kTableWords;
    lut_load<C>(lut[g], lane, [&](int i, uint32_t w) { return __ldg(tbl + i * kTableWords + w); });
  }
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      uint32_t y[C], m[Lut<C>::kMixed];
#pragma unroll
      for (int i = 0; i < C; ++i) y[i] = w == 0 ? x[i][v].x : w == 1 ? x[i][v].y : w == 2 ? x[i][v].z : x[i][v].w;
      lut_index<C>(y, m);
#pragma unroll
      for (int g = 0; g < NG; ++g)
        if (g == 0 || uint32_t(g) < groups) lut_mac<C>(lut[g], y, m, &acc[g][v][4 * w]);  // CTA-uniform
    }
}

// One tile = kApplyThreads threads x V 128-bit vectors of columns of job d,
// starting at byte tile_base (< d.vec_len).  NG = number of 4-output groups
// per pass over the inputs (outputs g*4 .. g*4+3).  Must be called by all
// kApplyThreads threads of the CTA (warp shuffles need full warps).
// ACC: outputs accumulate (dst ^= product) instead of being overwritten,
// for incremental parity updates (encode_single with i > 0, update).
// FEW: at most 2 inputs.
template <int NG, int V, bool VERIFY, bool ACC = false, bool FEW = false>
__device__ __forceinline__ void apply_tile(const uint8_t *const *ptrs, uint32_t *flags, const JobDesc &d,
                                           uint64_t tile_base) {
  const uint32_t lane = threadIdx.x & 31;
  // Thread column of vector v: tile_base + (v * kApplyThreads + tid) * 16, so a
  // warp's 32 loads of one vector cover 512 contiguous bytes.
  uint64_t col[V];
  bool active[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    col[v] = tile_base + (uint64_t(v) * kApplyThreads + threadIdx.x) * kApplyVec;
    active[v] = col[v] < d.vec_len;
  }
  const uint8_t *const *ptr = ptrs + d.ptr_off;
  const uint32_t n_in = d.n_in;
  for (uint32_t g0 = 0; g0 * 4 < d.n_out; g0 += NG) {
    const uint32_t groups = min(uint32_t(NG), (d.n_out + 3) / 4 - g0);
    uint32_t acc[NG][V][16];  // per column: 4 packed outputs
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[g][v][i] = 0;
    uint32_t j = 0;
#pragma unroll 1
    for (; !FEW && j + 5 <= n_in; j += 5) apply_step<5, NG, V>(ptr, d, g0, groups, j, col, active, lane, acc);
    const uint32_t left = n_in - j;  // CTA-uniform
    if (!FEW && left == 4)
      apply_step<3, NG, V, 1>(ptr, d, g0, groups, j, col, active, lane, acc);
    else if (!FEW && left == 3)
      apply_step<3, NG, V>(ptr, d, g0, groups, j, col, active, lane, acc);
    else if (left == 2)
      apply_step<1, NG, V, 1>(ptr, d, g0, groups, j, col, active, lane, acc);
    else if (left == 1)
      apply_step<1, NG, V>(ptr, d, g0, groups, j, col, active, lane, acc);
    bool bad = false;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        uint32_t o[4][4];  // [output r][word w]
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t tmp[4];
          transpose4(&acc[g][v][w * 4], tmp);
#pragma unroll
          for (int r = 0; r < 4; ++r) o[r][w] = tmp[r];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t out = (g0 + g) * 4 + r;
          if (out < d.n_out && active[v]) {
            uint8_t *dst = const_cast<uint8_t *>(ptr[n_in + out]) + col[v];
            if (VERIFY) {
              uint4 e = ld_stream(dst);
              bad |= (e.x != o[r][0]) | (e.y != o[r][1]) | (e.z != o[r][2]) | (e.w != o[r][3]);
              if (d.mode & kJobStore)
                st_stream(const_cast<uint8_t *>(ptr[n_in + d.n_out + out]) + col[v],
                          make_uint4(o[r][0], o[r][1], o[r][2], o[r][3]));
            } else if (ACC) {
              const uint4 e = *reinterpret_cast<const uint4 *>(dst);
              st_stream(dst, make_uint4(o[r][0] ^ e.x, o[r][1] ^ e.y, o[r][2] ^ e.z, o[r][3] ^ e.w));
            } else {
              st_stream(dst, make_uint4(o[r][0], o[r][1], o[r][2], o[r][3]));
            }
          }
        }
      }
    }
    if (VERIFY) {
      if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(flags + d.flag_idx, 1u);
    }
  }
}

// Byte-granular product of one column col (>= d.vec_len, < the shard length)
// of job d: the path for shard tails that are not a multiple of 16 bytes, or
// jobs whose pointers are not 16-byte aligned.  Returns true on a verify
// mismatch.
template <bool VERIFY, bool ACC = false>
__device__ __forceinline__ bool apply_column(const uint8_t *const *ptrs, const JobDesc &d, uint64_t col) {
  const uint8_t *const *ptr = ptrs + d.ptr_off;
  bool bad = false;
  for (uint32_t g = 0; g * 4 < d.n_out; ++g) {
    uint32_t acc = 0;
    // One loop in the two forms that compile to the shorter chain of loads:
    // 50+20 of 5001 bytes, encode 45 us in the first and 35 in the second,
    // verify 29 and 39.
    if (VERIFY) {
      for (uint32_t j = 0; j < d.n_in; ++j) {
        const uint32_t x = ptr[j][col];
        const uint32_t *tb = d.tbl + (g * d.n_in + j) * kTableWords;
        acc ^= __ldg(tb + (x & 15)) ^ __ldg(tb + 16 + (x >> 4));
      }
    } else {
      const uint32_t *tb = d.tbl + size_t(g) * d.n_in * kTableWords;
      for (uint32_t j = 0; j < d.n_in; ++j, tb += kTableWords) {
        const uint32_t x = ptr[j][col];
        acc ^= __ldg(tb + (x & 15)) ^ __ldg(tb + 16 + (x >> 4));
      }
    }
    for (uint32_t r = 0; r < 4 && g * 4 + r < d.n_out; ++r) {
      uint8_t *dst = const_cast<uint8_t *>(ptr[d.n_in + g * 4 + r]) + col;
      const uint8_t b = uint8_t(acc >> (8 * r));
      if (VERIFY) {
        bad |= (*dst != b);
        if (d.mode & kJobStore) const_cast<uint8_t *>(ptr[d.n_in + d.n_out + g * 4 + r])[col] = b;
      } else if (ACC)
        *dst ^= b;
      else
        *dst = b;
    }
  }
  return bad;
}

}  // namespace
}  // namespace rsgpu
