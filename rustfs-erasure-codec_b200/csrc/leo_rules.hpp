// leo_rules.hpp -- where the bit-sliced Leopard transforms are the faster ones.
// Plain host arithmetic, so that a test can compare the rules with measurements.
#pragma once

#include <cstdint>

#include "rsgpu.h"

namespace rsgpu {

// GF(2^8): whether operation op (RSGPU_OP_*) of a code (k data shards; m, n:
// transform sizes) on shards of len bytes, `columns` byte columns in all, is
// faster in the bit-sliced kernels (slice_fft.cuh) than in the register-stage
// ones (leo_fft.cuh).  Those use 4 columns a thread instead of 32 and narrow
// their tiles for short shards, so they win on little work; transforms of at
// most 16 lanes fit a thread's registers there and their data groups need no
// barriers, so they also win when k is many times m.  A rebuild of more than 8
// lanes is never slower here.  One B200, register-stage / bit-sliced, us, a
// launch among others:
//   encode 10+4   1 MiB columns 11 / 11, 2 MiB 17 / 17, 4 MiB 31 / 28, 16 MiB 125 / 84
//   encode 16+16  64 KiB 10 / 12, 256 KiB 10 / 12, 512 KiB 14 / 14, 1 MiB 25 / 19
//   verify 32+16  64 KiB 17 / 14 (encode 12 / 12), 1 MiB 39 / 33;  16+16 256 KiB 15 / 16
//   encode 17+17  64-byte shards 10 / 10, verify 14 / 12 (x 128);  verify 60+9 4 KiB 23 / 21
//   encode 64+32  64-byte shards x 256 16 / 21, 512-byte 21 / 14, 4 KiB x 16 21 / 17
//   encode 180+64 1 KiB x 32 27 / 31, 64 KiB 31 / 29, 256 KiB 94 / 43
//   verify 60+64  512 bytes 19 / 16, 16 KiB 19 / 16;  180+64 512 bytes x 64 31 / 31
//   encode 100+100  16 KiB 19 / 25, 56 KiB 27 / 27, 128 KiB 49 / 27, 256-byte x 256 27 / 37
//   rebuild 10+4  4 KiB 13 / 11, 256 KiB 15 / 10;  4+2 256 KiB 7.8 / 7.6, 1 MiB 14 / 10
inline bool slice_pays(int op, uint32_t k, uint32_t m, uint32_t n, uint64_t len, uint64_t columns) {
  if (op == RSGPU_OP_RECONSTRUCT) return n > 8 || columns >= (512u << 10);
  if (m < 16) return k <= 4 * m && columns >= (2u << 20);
  const bool verify = op == RSGPU_OP_VERIFY;
  if (m == 16) return k <= 64 && (columns >= (512u << 10) || (verify && k > 16));
  if (m == 32) return k <= 32 || len >= 512;
  return len >= 512 && (columns >= (56u << 10) || (verify && m == 64 && k <= 128));
}

// GF(2^16): the same for n_jobs stripes.  These kernels need 64 lanes to split
// and work on tiles of 2 KiB of a shard, which a length like 2112 fills to
// half; three launches a pass cost them some 20 us.  The register-stage kernels
// take one wave of 148 tiles of 128 to 512 bytes in about the time of one
// tile, and an encode's data groups one after another.  So encodes and verifies
// of few lanes go there up to one wave of columns (a single data group: two),
// and from four groups on only when the tiles are badly filled; the widest
// never.  One B200, register-stage / bit-sliced, us, a launch among others:
//   encode 60+64   64 KiB 17 / 24, 128 KiB 25 / 25, 256 KiB 45 / 33
//   encode 120+64  64 KiB 23 / 25, 128 KiB 35 / 29;  180+64 32 KiB 25 / 25 (verify 29 / 31), 128 KiB 47 / 37
//   encode 200+60  2 KiB 29 / 25, 2112 bytes x 64 55 / 61
//   encode 100+128 32 KiB 19 / 25, 64 KiB 27 / 27, 128 KiB 51 / 33
//   encode 200+128 32 KiB 25 / 26, 64 KiB 39 / 31, 2112 bytes x 32 39 / 45
//   encode 256+256 16 KiB 21 / 25, 32 KiB 39 / 29;  400+200 1 KiB x 4 29 / 27, x 16 29 / 31
//   encode 500+500 1 KiB 35 / 27, x 16 35 / 38, 2 KiB x 16 68 / 39, 1024+512 1 KiB x 8 51 / 35
//   encode 2048+1024 1 KiB 117 / 33, 16 KiB x 16 1882 / 858;  1024+512 16 KiB x 16 735 / 360
//   rebuild 40+16  1 KiB 39 / 23, 64+32 2 KiB x 4 43 / 25, 1024+512 16 KiB x 16 2412 / 1018
inline bool slice16_pays(int op, uint32_t k, uint32_t m, uint32_t n, uint64_t len, uint64_t n_jobs) {
  const uint64_t row = 2048, tiles = (len + row - 1) / row * n_jobs, columns = len * n_jobs;
  if (op == RSGPU_OP_RECONSTRUCT) return n >= 64 && len >= 1024;
  if (m < 64 || len < (m > 128 ? 1024 : 2048)) return false;
  if (m >= 1024) return true;
  const uint32_t groups = (k + m - 1) / m;
  const uint64_t wave = 148 * (m > 256 ? 128 : 32768 / m);
  if (m >= 256) return columns > wave || (tiles <= 8 && (groups > 1 || m == 512));
  return 3 * columns >= 2 * tiles * row && (groups > 3 || columns > (groups == 1 ? 2 : 1) * wave);
}

}  // namespace rsgpu
