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

}  // namespace rsgpu
