// slice_field.cuh -- bit-sliced arithmetic of the Leopard fields.
//
// 32 elements of a Leopard field are held as bit planes (plane b = bit b of
// all 32).  Multiplying by a constant is a GF(2)-linear map of those bits, so
// with the constant known at compile time it is a fixed network of plane XORs:
// no tables, no shuffles.
//
// Both fields are written in a Cantor basis (src/core/leopard_gf8/tables.rs:
// 8-145, src/core/leopard_gf16/tables.rs:8-116), whose first 4 (8) vectors
// span the subfield GF(16) (GF(256)).  The planes use the tower basis
// t_i = b_(i & 3) * [b_4 if i & 4] * [b_8 if i & 8] of the Cantor vectors b
// instead: it differs from the Cantor basis by a triangular map (applied once
// on load and once on store), and in it an element of GF(16) multiplies the
// 4-plane groups one by one.
//
// A constant is split into the nibbles of its tower coordinates, and each
// nibble selects one of 16 networks by a warp-uniform jump.  Nibble q's
// networks have about 2.1 * (1, 1.5, 2, 2.5)[q] terms a plane, and the
// transforms' constants are small in most layers (slice_fft.cuh).  One jump
// over the 256 constants of a byte was the alternative: the same number of
// XORs for the transforms' constants and sixteen times the code, which then
// would not stay in the instruction cache.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace rsgpu {
namespace {

template <int BITS>
struct CantorField;

template <>
struct CantorField<8> {
  static constexpr uint32_t kPoly = 0x11D;
  __host__ __device__ static constexpr uint32_t basis(int i) {
    constexpr uint32_t b[8] = {1, 214, 152, 146, 86, 200, 88, 230};
    return b[i];
  }
};
template <>
struct CantorField<16> {
  static constexpr uint32_t kPoly = 0x1002D;
  __host__ __device__ static constexpr uint32_t basis(int i) {
    constexpr uint32_t b[16] = {0x0001, 0xACCA, 0x3C0E, 0x163E, 0xC582, 0xED2E, 0x914C, 0x4012,
                                0x6C98, 0x10D8, 0x6A72, 0xB900, 0xFDB8, 0xFB34, 0xFF38, 0x991E};
    return b[i];
  }
};

// Polynomial-basis product.
template <int BITS>
__host__ __device__ constexpr uint32_t poly_mul(uint32_t a, uint32_t b) {
  uint32_t r = 0;
  for (int i = 0; i < BITS; ++i) {
    if ((b >> i) & 1) r ^= a;
    a <<= 1;
    if ((a >> BITS) & 1) a ^= CantorField<BITS>::kPoly;
  }
  return r;
}

// Inverse of the basis change: row i of coords() dotted with a polynomial
// gives Cantor coordinate i.
template <int BITS>
struct BasisInverse {
  uint32_t row[BITS];  // row[p]: coordinates of the polynomial x^p
};
template <int BITS>
__host__ __device__ constexpr BasisInverse<BITS> basis_inverse() {
  // Gauss-Jordan on the pairs (polynomial, coordinates) of the basis vectors.
  uint32_t poly[BITS] = {}, coord[BITS] = {};
  for (int i = 0; i < BITS; ++i) {
    poly[i] = CantorField<BITS>::basis(i);
    coord[i] = 1u << i;
  }
  BasisInverse<BITS> inv{};
  for (int p = 0; p < BITS; ++p) {
    int s = p;
    while (!((poly[s] >> p) & 1)) ++s;
    const uint32_t tp = poly[s], tc = coord[s];
    poly[s] = poly[p];
    coord[s] = coord[p];
    poly[p] = tp;
    coord[p] = tc;
    for (int i = 0; i < BITS; ++i)
      if (i != p && ((poly[i] >> p) & 1)) {
        poly[i] ^= tp;
        coord[i] ^= tc;
      }
  }
  for (int p = 0; p < BITS; ++p) inv.row[p] = coord[p];
  return inv;
}

template <int BITS>
__host__ __device__ constexpr uint32_t to_poly(uint32_t c) {
  uint32_t r = 0;
  for (int i = 0; i < BITS; ++i)
    if ((c >> i) & 1) r ^= CantorField<BITS>::basis(i);
  return r;
}
template <int BITS>
__host__ __device__ constexpr uint32_t to_coord(uint32_t p) {
  constexpr BasisInverse<BITS> inv = basis_inverse<BITS>();
  uint32_t r = 0;
  for (int i = 0; i < BITS; ++i)
    if ((p >> i) & 1) r ^= inv.row[i];
  return r;
}
template <int BITS>
__host__ __device__ constexpr uint32_t cantor_mul(uint32_t a, uint32_t b) {
  return to_coord<BITS>(poly_mul<BITS>(to_poly<BITS>(a), to_poly<BITS>(b)));
}

// Tower basis: vector i in Cantor coordinates, and the inverse change.
template <int BITS>
__host__ __device__ constexpr uint32_t tower_vec(int i) {
  uint32_t v = 1u << (i & 3);
  if (i & 4) v = cantor_mul<BITS>(v, 1u << 4);
  if (i & 8) v = cantor_mul<BITS>(v, 1u << 8);
  return v;
}
template <int BITS>
struct BasisPair {
  uint32_t to_cantor[BITS];  // Cantor coordinates of tower vector i
  uint32_t to_tower[BITS];   // tower coordinates of Cantor vector i
};
template <int BITS>
__host__ __device__ constexpr BasisPair<BITS> tower_basis() {
  // The change is unitriangular (vector i = Cantor vector i + lower ones), so
  // the inverse follows row by row.
  BasisPair<BITS> t{};
  for (int i = 0; i < BITS; ++i) {
    t.to_cantor[i] = tower_vec<BITS>(i);
    uint32_t r = 1u << i;
    for (int j = 0; j < i; ++j)
      if ((t.to_cantor[i] >> j) & 1) r ^= t.to_tower[j];
    t.to_tower[i] = r;
  }
  return t;
}
template <int BITS>
__host__ __device__ constexpr uint32_t cantor_to_tower(uint32_t c) {
  constexpr BasisPair<BITS> t = tower_basis<BITS>();
  uint32_t r = 0;
  for (int i = 0; i < BITS; ++i)
    if ((c >> i) & 1) r ^= t.to_tower[i];
  return r;
}
template <int BITS>
__host__ __device__ constexpr uint32_t tower_to_cantor(uint32_t c) {
  constexpr BasisPair<BITS> t = tower_basis<BITS>();
  uint32_t r = 0;
  for (int i = 0; i < BITS; ++i)
    if ((c >> i) & 1) r ^= t.to_cantor[i];
  return r;
}
template <int BITS>
__host__ __device__ constexpr uint32_t tower_mul(uint32_t a, uint32_t b) {
  return cantor_to_tower<BITS>(cantor_mul<BITS>(tower_to_cantor<BITS>(a), tower_to_cantor<BITS>(b)));
}

// A linear map of the coordinates: image plane r is the XOR of the planes b
// whose col[b] has bit r.
template <int BITS>
struct PlaneMap {
  uint32_t col[BITS];
};
template <int BITS, uint32_t C>
__host__ __device__ constexpr PlaneMap<BITS> mul_map() {
  PlaneMap<BITS> m{};
  for (int b = 0; b < BITS; ++b) m.col[b] = tower_mul<BITS>(C, 1u << b);
  return m;
}

// x ^= C * y on planes.
template <int BITS, uint32_t C>
__device__ __forceinline__ void mac_const(uint32_t *x, const uint32_t *y) {
  constexpr PlaneMap<BITS> net = mul_map<BITS, C>();
#pragma unroll
  for (int r = 0; r < BITS; ++r) {
#pragma unroll
    for (int b = 0; b < BITS; ++b)
      if ((net.col[b] >> r) & 1) x[r] ^= y[b];
  }
}

// Cantor -> tower planes and back, in place: vector i only involves lower
// ones, so ascending order reads only planes that are not yet changed.
template <int BITS>
__device__ __forceinline__ void planes_to_tower(uint32_t *v) {
  constexpr BasisPair<BITS> t = tower_basis<BITS>();
#pragma unroll
  for (int r = 0; r < BITS; ++r)
#pragma unroll
    for (int b = r + 1; b < BITS; ++b)
      if ((t.to_tower[b] >> r) & 1) v[r] ^= v[b];
}
template <int BITS>
__device__ __forceinline__ void planes_to_cantor(uint32_t *v) {
  constexpr BasisPair<BITS> t = tower_basis<BITS>();
#pragma unroll
  for (int r = 0; r < BITS; ++r)
#pragma unroll
    for (int b = r + 1; b < BITS; ++b)
      if ((t.to_cantor[b] >> r) & 1) v[r] ^= v[b];
}

// x ^= (n << SH) * y, and the same for two pairs, for a warp-uniform nibble n
// (the networks of slice_net.cuh).
template <int BITS, int SH>
__device__ __forceinline__ void mac_nibble(uint32_t n, uint32_t *x0, const uint32_t *y0);
template <int BITS, int SH>
__device__ __forceinline__ void mac2_nibble(uint32_t n, uint32_t *x0, const uint32_t *y0, uint32_t *x1,
                                            const uint32_t *y1);
// The same for half the planes of GF(2^16) and a constant of its subfield
// GF(256).
template <int SH>
__device__ __forceinline__ void sub_nibble(uint32_t n, uint32_t *x0, const uint32_t *y0);
template <int SH>
__device__ __forceinline__ void sub2_nibble(uint32_t n, uint32_t *x0, const uint32_t *y0, uint32_t *x1,
                                            const uint32_t *y1);
#include "slice_net.cuh"

// x ^= c * y in GF(2^8) for a warp-uniform constant in tower coordinates.
__device__ __forceinline__ void mac8(uint32_t c, uint32_t *x, const uint32_t *y) {
  mac_nibble<8, 0>(c & 15, x, y);
  mac_nibble<8, 4>((c >> 4) & 15, x, y);
}
// Tower coordinates of a Cantor constant, nibble by nibble.
template <int BITS>
struct NibbleTower {
  uint16_t v[BITS / 4][16];
};
template <int BITS>
__host__ __device__ constexpr NibbleTower<BITS> nibble_tower() {
  NibbleTower<BITS> t{};
  for (int q = 0; q < BITS / 4; ++q)
    for (uint32_t n = 0; n < 16; ++n) t.v[q][n] = uint16_t(cantor_to_tower<BITS>(n << (4 * q)));
  return t;
}
__constant__ const NibbleTower<8> c_tower8 = nibble_tower<8>();
__constant__ const NibbleTower<16> c_tower16 = nibble_tower<16>();
template <int BITS>
__device__ __forceinline__ uint32_t tower_const(uint32_t e) {
  if (BITS == 8) return c_tower8.v[0][e & 15] ^ c_tower8.v[1][e >> 4];
  return c_tower16.v[0][e & 15] ^ c_tower16.v[1][(e >> 4) & 15] ^ c_tower16.v[2][(e >> 8) & 15] ^
         c_tower16.v[3][e >> 12];
}

// The fields of the 8-plane transforms (slice_fft.cuh): Leopard GF(2^8), and
// half the planes of GF(2^16) under its subfield GF(256).
struct Gf8 {
  __device__ __forceinline__ static uint32_t tower(uint32_t e) { return tower_const<8>(e); }
  __device__ __forceinline__ static void mac(uint32_t c, uint32_t *x, const uint32_t *y) { mac8(c, x, y); }
  __device__ __forceinline__ static void mac2(uint32_t c, uint32_t *x0, const uint32_t *y0, uint32_t *x1,
                                              const uint32_t *y1) {
    mac2_nibble<8, 0>(c & 15, x0, y0, x1, y1);
    mac2_nibble<8, 4>(c >> 4, x0, y0, x1, y1);
  }
  __device__ __forceinline__ static void beta1(uint32_t *x, const uint32_t *y) { mac_const<8, 2>(x, y); }
};
struct Sub16 {
  __device__ __forceinline__ static uint32_t tower(uint32_t e) {
    return c_tower16.v[0][e & 15] ^ c_tower16.v[1][e >> 4];
  }
  __device__ __forceinline__ static void mac(uint32_t c, uint32_t *x, const uint32_t *y) {
    sub_nibble<0>(c & 15, x, y);
    sub_nibble<4>(c >> 4, x, y);
  }
  __device__ __forceinline__ static void mac2(uint32_t c, uint32_t *x0, const uint32_t *y0, uint32_t *x1,
                                              const uint32_t *y1) {
    sub2_nibble<0>(c & 15, x0, y0, x1, y1);
    sub2_nibble<4>(c >> 4, x0, y0, x1, y1);
  }
  __device__ __forceinline__ static void beta1(uint32_t *x, const uint32_t *y) {
    constexpr PlaneMap<16> net = mul_map<16, 2>();  // closed on the first 8 planes
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if ((net.col[b] >> r) & 1) x[r] ^= y[b];
  }
};

// Bytes of 8 words -> 8 bit planes, and back: the three swaps exchange one
// bit of the word index with one bit of the bit index each, so the map is its
// own inverse.  Which column a plane bit stands for is the same on the way in
// and out, and nothing in between depends on it.
__device__ __forceinline__ void slice_swap(uint32_t &a, uint32_t &b, uint32_t mask, int sh) {
  const uint32_t lo = (a & mask) | ((b << sh) & ~mask);
  b = ((a >> sh) & mask) | (b & ~mask);
  a = lo;
}
__device__ __forceinline__ void slice8(uint32_t *w) {
#pragma unroll
  for (int i = 0; i < 4; ++i) slice_swap(w[i], w[i + 4], 0x0F0F0F0Fu, 4);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (!(i & 2)) slice_swap(w[i], w[i + 2], 0x33333333u, 2);
#pragma unroll
  for (int i = 0; i < 8; i += 2) slice_swap(w[i], w[i + 1], 0x55555555u, 1);
}

}  // namespace
}  // namespace rsgpu
