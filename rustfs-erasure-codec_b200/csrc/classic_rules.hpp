// classic_rules.hpp -- which K1 kernel takes misaligned jobs, and verifies of
// few inputs.  Plain host arithmetic, so that a test can compare the rules with
// measurements.
#pragma once

#include <cstdint>

namespace rsgpu {

constexpr uint32_t kWordTile = 4096;  // columns of a work item of k_apply_unaligned

// Whether misaligned jobs of len bytes, n_jobs of them with up to max_out
// outputs, are faster by words (k_apply_unaligned) than one thread a byte
// column (k_apply_tail).  A word tile takes about as long with few columns as
// with 4096, and outputs in fours one after another, so the byte kernel wins
// while it has few columns a thread, and when the tiles are badly filled.  One
// B200, bytes / words, us:
//   encode 10+4  312 KiB of columns 10 / 12, 781 KiB 15 / 12, 1.25 MiB 21 / 16
//   encode 12+4  2.5 MiB in shards of 5001 bytes 41 / 39;  16+4 514 KiB of 1029 14 / 16
//   encode 10+6  488 KiB 15 / 19, 1.25 MiB 32 / 24
//   rebuild 50+20 781 KiB 92 / 127, 1.25 MiB 169 / 161, of 5001 bytes 172 / 248
//   verify 12+4  195 KiB 10 / 12, 312 KiB 12 / 12, 781 KiB 18 / 14
//   verify 50+20 312 KiB 82 / 119, 781 KiB of 5001 bytes 151 / 208, 1.25 MiB 258 / 208
inline bool words_pay(bool verify, uint32_t max_out, uint64_t len, uint64_t n_jobs) {
  const uint64_t words = len >= 12 ? (len - 8) / 4 : 0, columns = len * n_jobs;
  uint64_t padded = (words * 4 + kWordTile - 1) / kWordTile * kWordTile * n_jobs;
  if (!words) padded = uint64_t(kWordTile) * n_jobs;
  if (max_out > 4) return columns >= ((verify ? 512u : 1024u) << 10) && 8 * columns >= 5 * padded;
  return columns >= ((verify ? 256u : 704u) << 10) && 5 * columns >= 2 * padded;
}

// The same for launches that add to their outputs (n_in inputs: the changed
// shards of an update).  The word kernel reads and writes each output word
// between the others' bytes, so it needs inputs enough to pay for that: five, or
// as many as there are outputs beyond four, and a few rounds of tiles.  One B200,
// whole calls, bytes / words, us, shards of 4 MiB and of 16 MiB less 3 bytes:
//   10+4 encode_single 43 / 70, 145 / 192;  update of 3: 65 / 80, 278 / 299,
//   of 5: 78 / 88, 410 / 317, of 10: 145 / 109, 670 / 375
//   50+20 of 10: 458 / 517, of 20: 724 / 679, of 50: 1751 / 1238 (1 MiB 474 / 425)
inline bool words_pay_update(uint32_t n_in, uint32_t max_out, uint64_t len, uint64_t n_jobs) {
  return n_in >= 5 && (max_out <= 4 || n_in >= max_out) && n_in * len * n_jobs >= (32u << 20);
}

// Whether a verify of n_in inputs a job runs in the staged tile rather than with
// its tables in registers.  One or two inputs have next to no lookups to share,
// and the register tile keeps fewer of their bytes on the way (every stage has
// room for four parity shards).  One B200, staged / in registers, us:
//   verify 1+1  4 KiB x 1024 12 / 11, 64 KiB x 64 8.4 / 10, 1 MiB x 256 200 / 225
//   verify 2+1  1 KiB x 1024 14 / 10, 16 KiB x 64 8 / 8, 1 MiB x 64 71 / 75
//   verify 3+2  1 MiB x 64 90 / 86
inline bool verify_staged(uint32_t n_in, uint64_t len, uint64_t n_jobs) {
  return n_in <= 2 && len >= (16u << 10) && len * n_jobs >= (4u << 20);
}

}  // namespace rsgpu
