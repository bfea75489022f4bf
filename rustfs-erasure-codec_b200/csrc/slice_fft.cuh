// slice_fft.cuh -- Leopard GF(2^8) transforms on bit planes, one column tile
// at a time.
//
// A warp works on one lane (shard) group of a tile: each thread holds 32
// columns of a lane as 8 planes (32 bytes of the shard), so a butterfly of 32
// threads is 32 * 32 byte columns wide and its constant is warp-uniform.  Rows
// of all lanes live in shared memory, plane words of a thread as two 16-byte
// halves ([row][half][thread], so every access is a conflict-free 128-bit
// one); a pass runs two transform layers (radix 4) on four lanes held in
// registers.
//
// Constants.  The field's skew entry of a butterfly whose block starts at lane
// r with distance d is the element with Cantor coordinates (r + off) / d, off
// = the transform's first lane position (encoder IFFT of data group g:
// m + g * m, everything else: 0).  A radix-4 group at r needs e = (r + off) / d
// for its two inner blocks -- the second one's constant is e ^ 2, i.e. one
// fixed multiplication by b_1 on top -- and (r + off) / 2d for the outer one,
// so a group makes two warp-uniform constant selections for four butterflies
// (src/core/leopard_gf8/encode.rs:194-372, decode.rs:291-420; ops in
// src/core/leopard_gf16/ops.rs:375-511).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "apply_tile.cuh"
#include "leo_types.hpp"
#include "slice_field.cuh"

namespace rsgpu {
namespace {

// Inverse butterflies (IFFT): y ^= x; x ^= c * y.  Forward (FFT): x ^= c * y;
// y ^= x.
template <int BITS>
__device__ __forceinline__ void xor_planes(uint32_t *a, const uint32_t *b) {
#pragma unroll
  for (int i = 0; i < BITS; ++i) a[i] ^= b[i];
}
// Radix-4 on lanes r, r + d, r + 2d, r + 3d (e, e2: tower constants of the
// inner and the outer layer).
template <class F>
__device__ __forceinline__ void ifft4(uint32_t (*v)[8], uint32_t e, uint32_t e2) {
  xor_planes<8>(v[1], v[0]);
  xor_planes<8>(v[3], v[2]);
  F::mac2(e, v[0], v[1], v[2], v[3]);
  F::beta1(v[2], v[3]);
  xor_planes<8>(v[2], v[0]);
  xor_planes<8>(v[3], v[1]);
  F::mac2(e2, v[0], v[2], v[1], v[3]);
}
template <class F>
__device__ __forceinline__ void fft4(uint32_t (*v)[8], uint32_t e, uint32_t e2) {
  F::mac2(e2, v[0], v[2], v[1], v[3]);
  xor_planes<8>(v[2], v[0]);
  xor_planes<8>(v[3], v[1]);
  F::mac2(e, v[0], v[1], v[2], v[3]);
  F::beta1(v[2], v[3]);
  xor_planes<8>(v[1], v[0]);
  xor_planes<8>(v[3], v[2]);
}

__device__ __forceinline__ uint4 lds_words(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts_words(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Rows of a tile in shared memory: WT threads' words of a lane, two 16-byte
// halves each.  Threads past the row read its last thread's words and store
// nothing.
template <int WT>
struct Rows {
  static constexpr uint32_t kStride = WT * 32, kHalf = WT * 16;
  uint32_t base;  // this thread's words of row 0
  bool on;
  __device__ __forceinline__ Rows(uint32_t shared_base, uint32_t t)
      : base(shared_base + 16 * (WT < 32 ? min(t, uint32_t(WT - 1)) : t)), on(WT == 32 || t < WT) {}
  __device__ __forceinline__ uint32_t at(uint32_t row) const { return base + row * kStride; }
  __device__ __forceinline__ static void load(uint32_t addr, uint32_t *v) {
    const uint4 a = lds_words(addr), b = lds_words(addr + kHalf);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  }
  __device__ __forceinline__ void store(uint32_t addr, const uint32_t *v) const {
    if (!on) return;
    sts_words(addr, make_uint4(v[0], v[1], v[2], v[3]));
    sts_words(addr + kHalf, make_uint4(v[4], v[5], v[6], v[7]));
  }
  // Row r + j of a pass; a group that a pass skips.
  __device__ __forceinline__ void get(uint32_t r, uint32_t j, uint32_t *v) const { load(at(r) + j * kStride, v); }
  __device__ __forceinline__ void put(uint32_t r, uint32_t j, const uint32_t *v) const { store(at(r) + j * kStride, v); }
  __device__ __forceinline__ void skip(uint32_t, uint32_t) const {}
  __device__ __forceinline__ void store_xor(uint32_t addr, const uint32_t *v) const {
    uint32_t o[8];
    load(addr, o);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] ^= v[i];
    store(addr, o);
  }
};

// One pass of the transform over `lanes` rows of src; results go to dst
// (src itself, or with acc an accumulator they are XORed into).  Groups at or
// past `limit` are skipped, and so are groups none of whose 4-lane blocks is
// in `need` (bit i: lanes 4i..4i+3; ~0 for all).
template <int WT, bool FWD, class F = Gf8, class Src = Rows<WT>, class Dst = Rows<WT>>
__device__ __forceinline__ void slice_pass4(const Src &src, const Dst &dst, bool acc, uint32_t lanes, uint32_t lgd,
                                            uint32_t off, uint32_t limit, uint64_t need) {
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, d = 1u << lgd;
  const uint64_t block = d >= 64 ? ~0ull : (1ull << d) - 1;  // 4d lanes as bits of `need`
#pragma unroll 1
  for (uint32_t q = warp; q < (lanes >> 2); q += warps) {
    const uint32_t r = (q >> lgd) << (lgd + 2), l = r + (q & (d - 1));
    if (r >= limit || !((need >> (r >> 2)) & block)) {  // warp-uniform
      dst.skip(l, d);
      continue;
    }
    const uint32_t e = F::tower((r + off) >> lgd), e2 = F::tower((r + off) >> (lgd + 1));
    uint32_t v[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) src.get(l, j * d, v[j]);
    if (FWD)
      fft4<F>(v, e, e2);
    else
      ifft4<F>(v, e, e2);
    bool done = false;
    if constexpr (!FWD) {
      if (acc) {
#pragma unroll
        for (int j = 0; j < 4; ++j) dst.store_xor(dst.at(l) + j * (d * Rows<WT>::kStride), v[j]);
        done = true;
      }
    }
    if (!done) {
#pragma unroll
      for (int j = 0; j < 4; ++j) dst.put(l, j * d, v[j]);
    }
  }
}
// The leftover layer of an odd log2 size (the topmost one in both directions).
template <int WT, bool FWD, class F = Gf8>
__device__ __forceinline__ void slice_pass2(const Rows<WT> &src, const Rows<WT> &dst, bool acc, uint32_t lanes, uint32_t lgd,
                                            uint32_t off) {
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, d = 1u << lgd;
#pragma unroll 1
  for (uint32_t q = warp; q < (lanes >> 1); q += warps) {
    const uint32_t r = (q >> lgd) << (lgd + 1), l = r + (q & (d - 1));
    const uint32_t e = F::tower((r + off) >> lgd);
    uint32_t x[8], y[8];
    src.load(src.at(l), x);
    src.load(src.at(l + d), y);
    if (!FWD) xor_planes<8>(y, x);
    F::mac(e, x, y);
    if (FWD) xor_planes<8>(y, x);
    if (!FWD && acc) {
      dst.store_xor(dst.at(l), x);
      dst.store_xor(dst.at(l + d), y);
    } else {
      dst.store(dst.at(l), x);
      dst.store(dst.at(l + d), y);
    }
  }
}

// IFFT over 2^b lanes: radix-4 passes from distance 1 up.  The last pass XORs
// into dst when acc; with b == 0 there is no pass (the caller placed the row).
template <int WT, class F = Gf8>
__device__ __forceinline__ void slice_ifft(const Rows<WT> &src, const Rows<WT> &dst, bool acc, uint32_t b, uint32_t off,
                                           uint32_t limit) {
  uint32_t lgd = 0;
#pragma unroll 1
  for (; lgd + 2 <= b; lgd += 2) {
    const bool last = lgd + 2 == b;
    slice_pass4<WT, false, F>(src, last ? dst : src, last && acc, 1u << b, lgd, off, last ? ~0u : limit, ~0ull);
    __syncthreads();
  }
  if (lgd < b) {
    slice_pass2<WT, false, F>(src, dst, acc, 1u << b, lgd, off);
    __syncthreads();
  }
}
// FFT over 2^b lanes in place, from the top layer down.
template <int WT, class F = Gf8>
__device__ __forceinline__ void slice_fft(const Rows<WT> &s, uint32_t b, uint32_t limit, uint64_t need) {
  uint32_t lgd = b;
  if (b & 1) {
    slice_pass2<WT, true, F>(s, s, false, 1u << b, --lgd, 0);
    __syncthreads();
  }
#pragma unroll 1
  while (lgd >= 2) {
    lgd -= 2;
    slice_pass4<WT, true, F>(s, s, false, 1u << b, lgd, 0, limit, need);
    __syncthreads();
  }
}

// Formal derivative in place: lane l gains the XOR of the old lanes l | 2^t
// over the zero bits t of l (src/core/leopard_gf16/decode.rs:1100-1116).  A
// warp takes half the planes (one 16-byte half) of G consecutive lanes: the
// low bits come from its registers, the others from G loads a bit.  A lane
// depends only on lanes above it, and a round takes the groups in ascending
// order, reads everything, waits for the CTA, then writes.
template <int LG, int WT>
__device__ __forceinline__ void slice_derivative(const Rows<WT> &s, uint32_t n) {
  constexpr uint32_t G = 1u << LG;
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t items = (n >> LG) * 2;
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < items; i0 += warps) {
    // Warps past the last item redo it and store nothing.
    const uint32_t it = min(i0 + warp, items - 1), R = (it >> 1) << LG;
    const uint32_t base = s.at(R) + (it & 1) * Rows<WT>::kHalf;
    uint32_t v[G][4];
#pragma unroll
    for (uint32_t j = 0; j < G; ++j) {
      const uint4 u = lds_words(base + j * Rows<WT>::kStride);
      v[j][0] = u.x, v[j][1] = u.y, v[j][2] = u.z, v[j][3] = u.w;
    }
    // Ascending: v[j] gains only lanes above j, still unchanged.
#pragma unroll
    for (uint32_t j = 0; j < G; ++j)
#pragma unroll
      for (uint32_t t = 1; t < G; t <<= 1)
        if (!(j & t)) xor_planes<4>(v[j], v[j | t]);
#pragma unroll 1
    for (uint32_t t = G; t < n; t <<= 1) {
      if (R & t) continue;  // warp-uniform
      const uint32_t src = base + t * Rows<WT>::kStride;
#pragma unroll
      for (uint32_t j = 0; j < G; ++j) {
        const uint4 u = lds_words(src + j * Rows<WT>::kStride);
        v[j][0] ^= u.x, v[j][1] ^= u.y, v[j][2] ^= u.z, v[j][3] ^= u.w;
      }
    }
    __syncthreads();
    if (i0 + warp < items && s.on) {
#pragma unroll
      for (uint32_t j = 0; j < G; ++j)
        sts_words(base + j * Rows<WT>::kStride, make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]));
    }
    __syncthreads();
  }
}

// A thread's 32 columns of a shard: 16 bytes of each half of the tile, so a
// warp's accesses are contiguous.
template <int WT>
struct Cols {
  uint64_t a, b;
  bool on_a, on_b;
  __device__ __forceinline__ Cols(uint64_t tile, uint32_t t, uint64_t len) {
    a = tile + 16ull * t;
    b = a + 16 * WT;
    on_a = t < WT && a < len;
    on_b = t < WT && b < len;
  }
  __device__ __forceinline__ void load(const uint8_t *p, uint32_t *w) const {
    uint4 x = make_uint4(0, 0, 0, 0), y = x;
    if (on_a) x = ld_stream(p + a);
    if (on_b) y = ld_stream(p + b);
    w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
    w[4] = y.x, w[5] = y.y, w[6] = y.z, w[7] = y.w;
  }
  __device__ __forceinline__ void store(uint8_t *p, const uint32_t *w) const {
    if (on_a) st_stream(p + a, make_uint4(w[0], w[1], w[2], w[3]));
    if (on_b) st_stream(p + b, make_uint4(w[4], w[5], w[6], w[7]));
  }
};

// Encode one tile (with VERIFY: compare with the parity shards; returns this
// thread's mismatch).  Rows: the accumulator's m, then the scratch m of the
// data groups after the first.
template <int WT, bool VERIFY>
__device__ __forceinline__ uint32_t slice_encode_tile(uint32_t smem, const SliceArgs &a, const uint8_t *const *ptr,
                                                      uint64_t tile, uint64_t len) {
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, t = threadIdx.x & 31;
  const uint32_t m = a.m, k = a.k, b = 31 - __clz(m);
  const Rows<WT> acc(smem, t), tmp(smem + m * Rows<WT>::kStride, t);
  const Cols<WT> cols(tile, t, len);
#pragma unroll 1
  for (uint32_t g = 0; g * m < k; ++g) {
    const uint32_t cnt = min(m, k - g * m);
    const Rows<WT> &dst = (g && b) ? tmp : acc;
#pragma unroll 1
    for (uint32_t i = warp; i < m; i += warps) {
      uint32_t w[8];
      if (i < cnt) {
        cols.load(ptr[g * m + i], w);
        if (b) {  // one parity shard is the plain XOR of the data
          slice8(w);
          planes_to_tower<8>(w);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = 0;
      }
      if (g && !b)
        dst.store_xor(dst.at(i), w);
      else
        dst.store(dst.at(i), w);
    }
    __syncthreads();
    slice_ifft(dst, acc, g != 0, b, m + g * m, cnt);
  }
  slice_fft(acc, b, a.p, ~0ull);
  uint32_t mismatch = 0;
#pragma unroll 1
  for (uint32_t i = warp; i < a.p; i += warps) {
    uint32_t w[8];
    acc.load(acc.at(i), w);
    if (b) {
      planes_to_cantor<8>(w);
      slice8(w);
    }
    uint8_t *out = const_cast<uint8_t *>(ptr[k + i]);
    if (VERIFY) {
      uint32_t have[8];
      cols.load(out, have);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < 4 ? cols.on_a : cols.on_b) mismatch |= have[j] ^ w[j];
    } else {
      cols.store(out, w);
    }
  }
  return mismatch;
}

// What a decode tile needs of each lane, 9 bytes in shared memory: its shard
// pointer (16-byte aligned; bit 0 set: present, bit 1: target, 0: neither) and
// the tower constant of its locator (target: of the inverse locator).
struct LaneInfo {
  uint64_t *ptr;
  uint8_t *c;
  static constexpr uint32_t kBytes = 9;
};

// Fills a job's lane table (lane l: parity l, or data l - m) and the bits of
// the 4-lane blocks that hold a target, 8 blocks a byte.
__device__ __forceinline__ void slice_lane_info(const SliceArgs &a, const LeoJob &jd, LaneInfo info, uint8_t *need) {
  for (uint32_t l = threadIdx.x; l < ((a.n + 31) & ~31u); l += blockDim.x) {
    uint64_t ptr = 0;
    uint32_t c = 0;
    if (l < a.p || (l >= a.m && l < a.m + a.k)) {
      const uint32_t sh = l < a.p ? a.k + l : l - a.m;
      const uint32_t role = jd.role[sh];  // 1 present, 2 target
      if (role) {
        ptr = reinterpret_cast<uint64_t>(a.ptrs[jd.ptr_off + sh]) | role;
        c = a.elem[role == 1 ? jd.err[l] : a.mod - jd.err[l]];
      }
    }
    const uint32_t targets = __ballot_sync(0xffffffffu, (ptr & 2) != 0);
    if (l < a.n) {
      info.ptr[l] = ptr;
      info.c[l] = uint8_t(c);
    }
    if ((l & 31) == 0) {
      uint32_t bits = 0;
      for (int q = 0; q < 8; ++q) bits |= ((targets >> (4 * q)) & 15) ? 1u << q : 0;
      need[l >> 5] = uint8_t(bits);
    }
  }
}

// The middle of a decode over n = 2^b lanes, b >= 4, in place: the two highest
// IFFT layers, the formal derivative (src/core/leopard_gf16/decode.rs:
// 1100-1116: lane l gains the lanes l | 2^t over its zero bits t) and the two
// highest FFT layers, on lanes a, a + n/4, a + n/2, a + 3n/4.  With V the rows
// before, W = IFFT_top(V) and N_low, N_top the derivative's parts over the low
// bits and the top two,
//   FFT_top(W + N_top W + N_low W) = FFT_top((1 + N_top) IFFT_top V) + N_low V,
// because the FFT undoes the IFFT and acts on every a alike.  The block is the
// transform's first, so all its constants are fixed.  A row depends on rows of
// the same or a larger a, so with a taken in ascending rounds each round reads
// everything, waits for the CTA, then writes.
template <int WT, class F = Gf8>
__device__ __forceinline__ void slice_middle(const Rows<WT> &s, uint32_t n) {
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, items = n >> 2;
  const uint32_t quarter = items * Rows<WT>::kStride;
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < items; i0 += warps) {
    const uint32_t a = min(i0 + warp, items - 1);  // past the last: redone, not stored
    const uint32_t base = s.at(a);
    uint32_t v[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) Rows<WT>::load(base + j * quarter, v[j]);
    xor_planes<8>(v[1], v[0]);  // IFFT_top
    xor_planes<8>(v[3], v[2]);
    F::beta1(v[2], v[3]);
    xor_planes<8>(v[2], v[0]);
    xor_planes<8>(v[3], v[1]);
    xor_planes<8>(v[0], v[1]);  // 1 + N_top
    xor_planes<8>(v[0], v[2]);
    xor_planes<8>(v[1], v[3]);
    xor_planes<8>(v[2], v[3]);
    xor_planes<8>(v[2], v[0]);  // FFT_top
    xor_planes<8>(v[3], v[1]);
    F::beta1(v[2], v[3]);
    xor_planes<8>(v[1], v[0]);
    xor_planes<8>(v[3], v[2]);
#pragma unroll 1
    for (uint32_t t = 1; t < items; t <<= 1) {
      if (a & t) continue;  // warp-uniform
      const uint32_t src = base + t * Rows<WT>::kStride;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t u[8];
        Rows<WT>::load(src + j * quarter, u);
        xor_planes<8>(v[j], u);
      }
    }
    __syncthreads();
    if (i0 + warp < items) {
#pragma unroll
      for (int j = 0; j < 4; ++j) s.store(base + j * quarter, v[j]);
    }
    __syncthreads();
  }
}

// Reconstruct one tile: present lanes scaled by their locators, IFFT, formal
// derivative, FFT, targets scaled by the inverse locators.  info holds the
// job's lanes and need the 4-lane blocks that hold a target.  From 16 lanes on
// the first two layers take their lanes straight from the shards (four shards'
// loads in flight), the middle is one pass and the last two layers give theirs
// straight to the targets: 128+64 at 512 KiB x 16, 32 lost, 2218 -> 1950 us.
// The encode keeps a load and a store pass of its own: fused the same way, its
// small CTAs waited for instructions (32+16 encode 663 -> 693 us).
template <int WT>
__device__ __forceinline__ void slice_decode_tile(uint32_t smem, const SliceArgs &a, LaneInfo info, const uint8_t *need,
                                                  uint32_t input_count, uint64_t tile, uint64_t len) {
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, t = threadIdx.x & 31;
  const uint32_t n = a.n, b = 31 - __clz(n);
  const Rows<WT> s(smem, t);
  const Cols<WT> cols(tile, t, len);
  if (b >= 4) {
#pragma unroll 1
    for (uint32_t q = warp; q < (n >> 2); q += warps) {
      const uint32_t r = 4 * q;
      uint32_t v[4][8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j][i] = 0;
        const uint64_t ptr = info.ptr[r + j];
        if (ptr & 1) cols.load(reinterpret_cast<const uint8_t *>(ptr - 1), v[j]);  // warp-uniform
      }
      if (r < input_count) {
        // Four rounds over one copy of the networks, the lanes rotating
        // through v[0].
#pragma unroll 1
        for (uint32_t j = 0; j < 4; ++j) {
          uint32_t x[8] = {};
          if (info.ptr[r + j] & 1) {  // warp-uniform
            slice8(v[0]);
            planes_to_tower<8>(v[0]);
            mac8(info.c[r + j], x, v[0]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[0][i] = v[1][i];
            v[1][i] = v[2][i];
            v[2][i] = v[3][i];
            v[3][i] = x[i];
          }
        }
        ifft4<Gf8>(v, tower_const<8>(r), tower_const<8>(r >> 1));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) s.store(s.at(r + j), v[j]);
    }
    __syncthreads();
    // Layers 2 .. b - 3: for an odd b the first of them alone.
    uint32_t lgd = 2;
    if (b & 1) {
      slice_pass2<WT, false>(s, s, false, n, lgd++, 0);
      __syncthreads();
    }
#pragma unroll 1
    for (; lgd < b - 2; lgd += 2) {
      slice_pass4<WT, false>(s, s, false, n, lgd, 0, input_count, ~0ull);
      __syncthreads();
    }
    slice_middle<WT>(s, n);
    const uint64_t blocks = *reinterpret_cast<const uint64_t *>(need);
    const uint32_t limit = a.m + a.k;
#pragma unroll 1
    while (lgd > 2 + (b & 1)) {
      lgd -= 2;
      slice_pass4<WT, true>(s, s, false, n, lgd, 0, limit, blocks);
      __syncthreads();
    }
    if (b & 1) {
      slice_pass2<WT, true>(s, s, false, n, 2, 0);
      __syncthreads();
    }
#pragma unroll 1
    for (uint32_t q = warp; q < (n >> 2); q += warps) {
      const uint32_t r = 4 * q;
      if (!((blocks >> q) & 1)) continue;  // warp-uniform
      uint32_t v[4][8];
#pragma unroll
      for (int j = 0; j < 4; ++j) Rows<WT>::load(s.at(r + j), v[j]);
      fft4<Gf8>(v, tower_const<8>(r), tower_const<8>(r >> 1));
#pragma unroll 1
      for (uint32_t j = 0; j < 4; ++j) {
        const uint64_t ptr = info.ptr[r + j];
        if (ptr & 2) {  // warp-uniform
          uint32_t x[8] = {};
          mac8(info.c[r + j], x, v[0]);
          planes_to_cantor<8>(x);
          slice8(x);
          cols.store(reinterpret_cast<uint8_t *>(ptr - 2), x);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          v[0][i] = v[1][i];
          v[1][i] = v[2][i];
          v[2][i] = v[3][i];
        }
      }
    }
    return;
  }
#pragma unroll 1
  for (uint32_t i = warp; i < n; i += warps) {
    uint32_t x[8] = {};
    const uint64_t ptr = info.ptr[i];
    if (ptr & 1) {  // warp-uniform
      uint32_t y[8];
      cols.load(reinterpret_cast<const uint8_t *>(ptr - 1), y);
      slice8(y);
      planes_to_tower<8>(y);
      mac8(info.c[i], x, y);
    }
    s.store(s.at(i), x);
  }
  __syncthreads();
  slice_ifft(s, s, false, b, 0, input_count);
  if (n >= 8)
    slice_derivative<3>(s, n);
  else if (n == 4)
    slice_derivative<2>(s, n);
  else
    slice_derivative<1>(s, n);
  slice_fft(s, b, a.m + a.k, *reinterpret_cast<const uint64_t *>(need));
#pragma unroll 1
  for (uint32_t i = warp; i < n; i += warps) {
    const uint64_t ptr = info.ptr[i];
    if (!(ptr & 2)) continue;  // warp-uniform
    uint32_t y[8], x[8] = {};
    s.load(s.at(i), y);
    mac8(info.c[i], x, y);
    planes_to_cantor<8>(x);
    slice8(x);
    cols.store(reinterpret_cast<uint8_t *>(ptr - 2), x);
  }
}

}  // namespace
}  // namespace rsgpu
