// leo_slice.hpp -- host side of the bit-sliced Leopard GF(2^8) transforms.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "leo_rules.hpp"
#include "leo_types.hpp"

namespace rsgpu {

struct SliceShape {
  int grid = 0, threads = 0;
  size_t smem = 0;
};
// Fills the tile width and rows of `a` (its geometry, len and n_jobs set) and
// the launch shape of operation op (RSGPU_OP_*).
int slice_configure(int op, SliceArgs &a, SliceShape &sh);
uint64_t slice_tile_bytes(int op, uint32_t k, uint32_t m, uint32_t n);
int slice_launch(int op, const SliceArgs &a, const SliceShape &sh, cudaStream_t s);
// Tower coordinates of the element of each log value of the 8- or 16-bit
// field, from its exp table.
void slice_elements(int bits, const uint16_t *exp, uint32_t order, uint16_t *out);

// Scratch a GF(2^16) launch may use in the codec's slab, and in a buffer of
// its stream (the request server keeps one per stream).  Waves of work items
// matter more than keeping the rows in L2: 1024+512 at 16 KiB x 16 rebuilds in
// 1391 us with 96 MiB, 1302 with 256, 1161 with 900 (every tile at once),
// encodes in 567, 556 and 523.
constexpr uint64_t kSlabScratch16 = uint64_t(256) << 20, kStreamScratch16 = uint64_t(96) << 20;
// Launches that need up to this have rows of their own instead: about where a
// launch fills the GPU by itself (1024+512 encode of one 16 KiB stripe, 25 MiB),
// so that larger ones lose nothing by running one after another.
constexpr uint64_t kOwnRows16 = uint64_t(32) << 20;
// GF(2^16).  Fills the split and tile counts of `a` (its geometry, len, n_jobs
// and max_scratch set); false when the code or shard length is not covered.
bool slice16_configure(int op, Slice16Args &a);
// Scratch bytes of a launch over `tiles` column tiles (bounded: wider launches
// go in chunks).
size_t slice16_scratch_bytes(const Slice16Args &a, uint64_t tiles);
size_t slice16_scratch_limit(const Slice16Args &a);  // ... over any number of tiles
// Kernels of a launch, and the launch: `scratch` must hold
// slice16_scratch_bytes and is private to the launch until it has run.
uint64_t slice16_kernels(const Slice16Args &a);
int slice16_launch(int op, Slice16Args a, void *scratch, cudaStream_t s);

}  // namespace rsgpu
