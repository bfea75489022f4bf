// k_classic.cu -- sm_100a kernels of the classic Reed-Solomon path.
//
// K1 (matrix apply): out[r] = sum_j c[r][j] * in[j] over GF(2^8), bytewise,
//   for encode, reconstruct (composed recovery rows) and verify (compare
//   instead of store).  It replaces the reference's row dot-product loops
//   (src/core/encode.rs:532-602, src/galois_8/x86/gfni_rows.rs:15-288).  The
//   per-tile device code and its design notes are in apply_tile.cuh; this file
//   holds the grid-stride launches over one batch.
//
// K3 (decode tables): Gauss-Jordan inversion of the selected survivor rows,
//   composition of the requested parity rows and packing of the nibble
//   tables, one CTA per erasure pattern (src/core/reconstruct.rs:1068-1174,
//   src/core/recovery_plan.rs:425-517).
#include <cuda_runtime.h>

#include <cstdlib>

#include "apply_tile.cuh"
#include "classic_rules.hpp"
#include "common.hpp"
#include "kernels.hpp"
#include "launch_cfg.hpp"

namespace rsgpu {

namespace {

// The launch's jobs and pointer table; the arguments must be __grid_constant__,
// so that their address can be taken.
__device__ __forceinline__ const JobDesc *job_list(const ApplyArgs &a) { return a.jobs ? a.jobs : &a.job; }
__device__ __forceinline__ const uint8_t *const *ptr_list(const ApplyArgs &a) { return a.jobs ? a.ptrs : a.job_ptrs; }

// Grid-stride loop of apply_tile over every (job, tile) of a launch, inputs
// loaded straight into registers: the tile for more than 4 outputs and for
// accumulating (incremental parity) launches.
template <int NG, bool VERIFY, bool ACC, int MINB>
__global__ void __launch_bounds__(kApplyThreads, MINB) k_apply_vec(const __grid_constant__ ApplyArgs a) {
  const JobDesc *const jobs = job_list(a);
  const uint8_t *const *const ptrs = ptr_list(a);
  constexpr uint32_t kTile = kApplyThreads * kApplyVec;
  const uint32_t tiles_per_job = uint32_t((a.len + kTile - 1) / kTile);
  const uint32_t total = tiles_per_job * a.n_jobs;
  for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
    const uint32_t job = t / tiles_per_job;
    const uint64_t tile_base = uint64_t(t - job * tiles_per_job) * kTile;
    const JobDesc d = jobs[job];
    if (tile_base >= d.vec_len) continue;  // CTA-uniform
    apply_tile<NG, 1, VERIFY, ACC>(ptrs, a.flags, d, tile_base);
  }
}

// ------------------------------------------------------------------ K1, TMA-staged
// The product for at most 4 outputs with the input tiles staged in
// shared memory by the bulk-copy (TMA) unit: one producer warp streams each
// step's tile slices (one contiguous 256 * 16 * V-byte slice per input shard,
// cp.async.bulk with completion on the stage's mbarrier) into a ring of S
// stages of 4 slots; kApplyThreads consumer threads wait for a stage, run the
// table arithmetic from shared memory and release it.  A step is up to 4
// input shards of one tile, or for verify the tile's <= 4 parity shards.
// n_out <= 4 only.  Every wait is bounded (about 2 s of SM clock); a wait
// that runs out sets *a.stall (the codec's status word, read back by the
// next synchronous call as RSGPU_ERR_DEVICE_TIMEOUT), and the producer then
// waits, bounded again, for the copies it has in flight before it exits.
// Measured against inputs loaded straight to registers (32 bytes a thread, four
// inputs in flight, the same pairs of 16-entry lookups) on 1024 x 1 MiB stripes: 10+4 encode 4650 vs 4268 GB/s; global-load stalls per
// issued instruction fall from 4.1 to 1.7, and the bulk copies do not compete
// with the table shuffles for the L1 data pipe (cp.async staging, which
// does, was 7-14% slower than the register path).
constexpr long long kStallCycles = 4000000000ll;

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Wait for the completion of the barrier phase with this parity; false when
// the wait ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > kStallCycles) return false;
  }
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr)
               : "memory");
  return v;
}

template <int V, int S, bool VERIFY>
__global__ void __launch_bounds__(kApplyThreads + 32, 2) k_apply_tma(const __grid_constant__ ApplyArgs a) {
  const JobDesc *const jobs = job_list(a);
  const uint8_t *const *const ptrs = ptr_list(a);
  constexpr uint32_t kSlot = kApplyThreads * kApplyVec * V;  // one input's slice of a tile
  extern __shared__ __align__(128) uint8_t tma_smem[];
  __shared__ __align__(8) uint64_t full[S], empty[S];
  // The 4+4 nibble tables (words 0..31 of each input's packed table) of each
  // stage's inputs, copied with the data when the launch's jobs carry
  // different tables (a batch of stripes with different erasure patterns):
  // read from L2 after the stage's wait, they put an L2 round trip on every
  // step (10+4 rebuild 3.2 -> 4.2 TB/s).  A table that every job shares stays
  // L1-resident and is read with plain loads.
  __shared__ __align__(16) uint32_t tma_tbl[S][4][32];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t sbase = uint32_t(__cvta_generic_to_shared(tma_smem));
  const uint32_t tbase = uint32_t(__cvta_generic_to_shared(&tma_tbl[0][0][0]));
  const uint32_t fbar = uint32_t(__cvta_generic_to_shared(full));
  const uint32_t ebar = uint32_t(__cvta_generic_to_shared(empty));
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(fbar + 8 * s, 1);
      mbar_init(ebar + 8 * s, kApplyThreads / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const uint32_t tiles_per_job = uint32_t((a.len + kSlot - 1) / kSlot);
  const uint32_t total = tiles_per_job * a.n_jobs;

  if (tid >= kApplyThreads) {  // producer warp: one lane issues every copy
    if (tid != kApplyThreads) return;
    uint32_t it = 0;
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const uint32_t job = t / tiles_per_job;
      const uint64_t base = uint64_t(t - job * tiles_per_job) * kSlot;
      const JobDesc d = jobs[job];
      if (base >= d.vec_len) continue;
      const uint32_t valid = uint32_t(d.vec_len - base < kSlot ? d.vec_len - base : kSlot);
      const uint8_t *const *ptr = ptrs + d.ptr_off;
      const bool tbl_copy = a.tbl_stage && d.tbl && (reinterpret_cast<uintptr_t>(d.tbl) & 15) == 0;
      const uint32_t steps = (d.n_in + 3) / 4 + (VERIFY ? 1 : 0);
      for (uint32_t step = 0; step < steps; ++step, ++it) {
        const uint32_t s = it % S, ph = (it / S) & 1;
        if (!mbar_wait(ebar + 8 * s, ph ^ 1)) {
          ok = false;
          break;
        }
        const bool par = VERIFY && step * 4 >= d.n_in;
        const uint32_t j0 = par ? d.n_in : step * 4;
        const uint32_t rows = par ? d.n_out : min(4u, d.n_in - j0);
        const bool tbl_here = tbl_copy && !par;
        mbar_expect_tx(fbar + 8 * s, rows * valid + (tbl_here ? rows * 128 : 0));
        for (uint32_t b = 0; b < rows; ++b)
          bulk_load(sbase + (s * 4 + b) * kSlot, ptr[j0 + b] + base, valid, fbar + 8 * s);
        if (tbl_here)
          for (uint32_t b = 0; b < rows; ++b)
            bulk_load(tbase + (s * 4 + b) * 128, d.tbl + (j0 + b) * kTableWords, 128, fbar + 8 * s);
      }
    }
    if (!ok) {
      if (a.stall) atomicOr(a.stall, 1u);
      // Copies already issued land in stages the consumers stopped reading:
      // wait (bounded) for them before the CTA's shared memory goes away.
      for (uint32_t k = 0; k < S && k < it; ++k) {
        const uint32_t i = it - 1 - k;
        mbar_wait(fbar + 8 * (i % S), (i / S) & 1);
      }
    }
    return;
  }

  // Consumers: the same (tile, step) sequence as the producer.
  uint32_t it = 0;
  for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
    const uint32_t job = t / tiles_per_job;
    const uint64_t base = uint64_t(t - job * tiles_per_job) * kSlot;
    const JobDesc d = jobs[job];
    if (base >= d.vec_len) continue;
    const uint32_t n_in = d.n_in;
    const bool tbl_copy = a.tbl_stage && d.tbl && (reinterpret_cast<uintptr_t>(d.tbl) & 15) == 0;  // as the producer decides
    const uint32_t steps = (n_in + 3) / 4 + (VERIFY ? 1 : 0);
    uint64_t col[V];
    bool active[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      col[v] = base + (uint64_t(v) * kApplyThreads + tid) * kApplyVec;
      active[v] = col[v] < d.vec_len;
    }
    uint32_t acc[V][16];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int i = 0; i < 16; ++i) acc[v][i] = 0;
    bool bad = false;
    for (uint32_t step = 0; step < steps; ++step, ++it) {
      const uint32_t s = it % S, ph = (it / S) & 1;
      if (!mbar_wait(fbar + 8 * s, ph)) {
        if (a.stall) atomicOr(a.stall, 1u);
        return;
      }
      const uint32_t slot0 = sbase + s * 4 * kSlot + tid * kApplyVec;
      const bool par = VERIFY && step * 4 >= n_in;
      if (!par) {
        const uint32_t j0 = step * 4;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          if (j0 + b >= n_in) break;  // warp-uniform
          uint32_t lo, hi;
          if (tbl_copy) {
            const uint32_t ta = tbase + (s * 4 + b) * 128 + (lane & 15) * 4;
            lo = lds32(ta);
            hi = lds32(ta + 64);
          } else {
            const uint32_t *tb = d.tbl + (j0 + b) * kTableWords;
            lo = __ldg(tb + (lane & 15));
            hi = __ldg(tb + 16 + (lane & 15));
          }
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const uint4 x = lds128(slot0 + b * kSlot + v * kApplyThreads * kApplyVec);
            mac4(x.x, lo, hi, &acc[v][0]);
            mac4(x.y, lo, hi, &acc[v][4]);
            mac4(x.z, lo, hi, &acc[v][8]);
            mac4(x.w, lo, hi, &acc[v][12]);
          }
        }
      }
      if (step + 1 == steps) {  // outputs of this tile (parity rows are in this stage when VERIFY)
#pragma unroll
        for (int v = 0; v < V; ++v) {
          uint32_t o[4][4];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            uint32_t tmp[4];
            transpose4(&acc[v][w * 4], tmp);
#pragma unroll
            for (int r = 0; r < 4; ++r) o[r][w] = tmp[r];
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (uint32_t(r) < d.n_out && active[v]) {
              if (VERIFY) {
                const uint4 e = lds128(slot0 + r * kSlot + v * kApplyThreads * kApplyVec);
                bad |= (e.x != o[r][0]) | (e.y != o[r][1]) | (e.z != o[r][2]) | (e.w != o[r][3]);
                if (d.mode & kJobStore)
                  st_stream(const_cast<uint8_t *>(ptrs[d.ptr_off + n_in + d.n_out + r]) + col[v],
                            make_uint4(o[r][0], o[r][1], o[r][2], o[r][3]));
              } else {
                uint8_t *dst = const_cast<uint8_t *>(ptrs[d.ptr_off + n_in + r]) + col[v];
                st_stream(dst, make_uint4(o[r][0], o[r][1], o[r][2], o[r][3]));
              }
            }
          }
        }
        if (VERIFY && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags + d.flag_idx, 1u);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(ebar + 8 * s);
    }
  }
}

// ------------------------------------------------------------------ K1, tables in registers
// The product for at most 4 outputs over K <= kRegInputs inputs, all lookup
// tables of the K inputs in registers (8 per five inputs, see apply_tile.cuh),
// loaded when the CTA meets another table, so the loop over columns is nothing
// but data reads, shuffles and XORs.  What bounds it is the L1 data pipe: of
// about 8 wavefronts per input word (128 bytes a warp) 6.4 are shuffles, 1 is
// the data read.  The staged tile above needs 8 shuffles and re-reads two
// tables per input and step, in 96 registers; this one fits 72, so three CTAs
// share an SM and the shuffle latency is hidden (10+4 encode, 1 MiB x 512:
// 4498 -> 5351 GB/s while the clock is near its maximum, the pipe 81% busy; in
// long runs deep in the power cap 4045 -> 4560, 71% of the copy peak).
// A CTA takes a contiguous run of tiles: launches whose stripes carry
// different tables then change tables once per stripe, not once per tile.
// The producer warp, the mbarrier ring and its bounded waits are
// k_apply_tma's; a stage is one tile of all K inputs (for verify also the <= 4
// parity shards).
constexpr int kRegInputs = 20;

template <int K, bool VERIFY>
struct RegShape {
  static constexpr int kSlots = K + (VERIFY ? 4 : 0);
  // Words a thread reads at a time: two (64-bit reads) while they fit the
  // registers of three CTAs an SM.
  static constexpr int kWords = K <= 10 ? 2 : 1;
  // Bytes of every shard a tile: enough work between two barrier waits.  A
  // verify of 4 inputs stages 8 shards; at 8 KiB each one CTA would fill the SM
  // (4+2 1 MiB x 64 121 us; 107 at 4 KiB, as in the staged tile).
  static constexpr uint32_t kTile = K <= 4 - VERIFY ? 8192 : K <= 7 ? 4096 : 2048;
  static constexpr int kFit = int(74 * 1024 / (kSlots * kTile));
  static constexpr int kStages = kFit < 2 ? 2 : kFit > 4 ? 4 : kFit;
  static constexpr int kBlocks = kFit < 2 || K > 13 ? 2 : 3;
  static constexpr size_t kSmem = size_t(kStages) * kSlots * kTile;
};

template <int K, bool VERIFY>
__global__ void __launch_bounds__(kApplyThreads + 32, RegShape<K, VERIFY>::kBlocks) k_apply_reg(const __grid_constant__ ApplyArgs a) {
  const JobDesc *const jobs = job_list(a);
  const uint8_t *const *const ptrs = ptr_list(a);
  using Shape = RegShape<K, VERIFY>;
  constexpr int S = Shape::kStages, W = Shape::kWords;
  constexpr uint32_t kTile = Shape::kTile, kStageBytes = Shape::kSlots * kTile;
  extern __shared__ __align__(128) uint8_t reg_smem[];
  __shared__ __align__(8) uint64_t full[S], empty[S];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t sbase = uint32_t(__cvta_generic_to_shared(reg_smem));
  const uint32_t fbar = uint32_t(__cvta_generic_to_shared(full));
  const uint32_t ebar = uint32_t(__cvta_generic_to_shared(empty));
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(fbar + 8 * s, 1);
      mbar_init(ebar + 8 * s, kApplyThreads / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const uint32_t tiles_per_job = uint32_t((a.len + kTile - 1) / kTile);
  const uint64_t total = uint64_t(tiles_per_job) * a.n_jobs;
  const uint32_t t0 = uint32_t(total * blockIdx.x / gridDim.x), t1 = uint32_t(total * (blockIdx.x + 1) / gridDim.x);
  uint32_t job = t0 / tiles_per_job, tile = t0 - job * tiles_per_job;
  uint32_t s = 0, ph = 0;  // ring position and its phase

  if (tid >= kApplyThreads) {  // producer warp: one lane issues every copy
    if (tid != kApplyThreads) return;
    uint32_t issued = 0;
    bool ok = true;
    for (uint32_t t = t0; t < t1; ++t) {
      const JobDesc d = jobs[job];
      const uint64_t base = uint64_t(tile) * kTile;
      if (base < d.vec_len) {
        const uint32_t valid = uint32_t(d.vec_len - base < kTile ? d.vec_len - base : kTile);
        const uint32_t rows = K + (VERIFY ? d.n_out : 0);
        const uint8_t *const *ptr = ptrs + d.ptr_off;
        if (!mbar_wait(ebar + 8 * s, ph ^ 1)) {
          ok = false;
          break;
        }
        mbar_expect_tx(fbar + 8 * s, rows * valid);
        for (uint32_t b = 0; b < rows; ++b)
          bulk_load(sbase + s * kStageBytes + b * kTile, ptr[b] + base, valid, fbar + 8 * s);
        ++issued;
        if (++s == S) s = 0, ph ^= 1;
      }
      if (++tile == tiles_per_job) tile = 0, ++job;
    }
    if (!ok) {
      if (a.stall) atomicOr(a.stall, 1u);
      // Wait (bounded) for the copies in flight before the CTA's shared
      // memory goes away: the last min(S, issued) stages.
      for (uint32_t k = 0; k < S && k < issued; ++k) {
        if (s == 0) s = S, ph ^= 1;
        --s;
        mbar_wait(fbar + 8 * s, ph);
      }
    }
    return;
  }

  LutSet<K> lut;
  const uint32_t *cur = nullptr;
  JobDesc d{};
  uint8_t *dst[4];  // this job's outputs (verify: where verify_store puts them)
  bool fresh = true;
  for (uint32_t t = t0; t < t1; ++t) {
    const uint64_t base = uint64_t(tile) * kTile;
    if (fresh) {
      fresh = false;
      d = jobs[job];
      const uint8_t *const *out = ptrs + d.ptr_off + K + (VERIFY ? d.n_out : 0);
#pragma unroll
      for (int r = 0; r < 4; ++r)
        dst[r] = uint32_t(r) < d.n_out && (!VERIFY || (d.mode & kJobStore)) ? const_cast<uint8_t *>(out[r]) : nullptr;
      if (d.tbl != cur) {
        lut.load(d.tbl, lane);
        cur = d.tbl;
      }
    }
    if (base < d.vec_len) {
      if (!mbar_wait(fbar + 8 * s, ph)) {
        if (a.stall) atomicOr(a.stall, 1u);
        return;
      }
      bool bad = false;
#pragma unroll 1
      for (uint32_t sub = 0; sub < kTile / (kApplyThreads * 4 * W); ++sub) {
        if (base + sub * (kApplyThreads * 4 * W) >= d.vec_len) break;  // CTA-uniform
        const uint32_t off = (sub * kApplyThreads + tid) * 4 * W;
        const uint32_t slot = sbase + s * kStageBytes + off;
        uint32_t x[W][K], acc[W][4];
#pragma unroll
        for (int j = 0; j < K; ++j) {
          if (W == 2)
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(x[0][j]), "=r"(x[W - 1][j]) : "r"(slot + j * kTile) : "memory");
          else
            x[0][j] = lds32(slot + j * kTile);
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
          uint32_t o[4] = {0, 0, 0, 0};
          lut.mac(x[w], o);
          transpose4(o, acc[w]);
        }
        const uint64_t col = base + off;
        if (col < d.vec_len) {
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (VERIFY && uint32_t(r) < d.n_out) {
#pragma unroll
              for (int w = 0; w < W; ++w) bad |= lds32(slot + (K + r) * kTile + 4 * w) != acc[w][r];
            }
            if (dst[r]) {
              if (W == 2)
                asm volatile("st.global.L1::no_allocate.v2.u32 [%0], {%1,%2};" ::"l"(dst[r] + col), "r"(acc[0][r]),
                             "r"(acc[W - 1][r])
                             : "memory");
              else
                asm volatile("st.global.L1::no_allocate.u32 [%0], %1;" ::"l"(dst[r] + col), "r"(acc[0][r]) : "memory");
            }
          }
        }
      }
      if (VERIFY && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags + d.flag_idx, 1u);
      __syncwarp();
      if (lane == 0) mbar_arrive(ebar + 8 * s);
      if (++s == S) s = 0, ph ^= 1;
    }
    if (++tile == tiles_per_job) tile = 0, ++job, fresh = true;
  }
}

// Byte-granular path for the columns past each job's vec_len.  One thread per
// byte column.  INLINE: the job and its pointers are in the arguments; a choice
// made in the kernel made every read of them a generic one (50+20 encode of
// 5001-byte shards 37 -> 45 us).
template <bool VERIFY, bool ACC, bool INLINE>
__global__ void k_apply_tail(const __grid_constant__ ApplyArgs a, uint64_t max_tail) {
  const JobDesc *const jobs = INLINE ? &a.job : a.jobs;
  const uint8_t *const *const ptrs = INLINE ? a.job_ptrs : a.ptrs;
  const uint64_t n = max_tail * a.n_jobs;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t job = uint32_t(i / max_tail);
    const JobDesc d = jobs[job];
    const uint64_t col = d.vec_len + (i - uint64_t(job) * max_tail);
    if (col >= a.len || (d.mode & kJobUnaligned)) continue;
    if (apply_column<VERIFY, ACC>(ptrs, d, col) && VERIFY) atomicOr(a.flags + d.flag_idx, 1u);
  }
}

// ------------------------------------------------------------------ K1, any alignment
// Jobs whose pointers are not all 16-byte aligned (shards of odd length packed
// back to back, for one), any number of inputs and outputs.  A thread takes
// kWordsU words of four columns, 128 bytes of consecutive words a warp; an
// input word at an odd address is put together from the two aligned words
// around it, an output word is written as the aligned word that overlaps it
// most (its neighbour's bytes come by a shuffle) with single bytes at the ends
// of a warp's run.  The columns covered this way, 4 to 4 + 4 * n, keep every
// aligned word inside the shard; the few before and after are the work of an
// extra warp.  Against one thread a byte column (k_apply_tail, still the faster
// one on few columns: classic_rules.hpp): verify of 128 12+4 stripes of 100003
// bytes 351 -> 103 us, encode 264 -> 115, 24+4 at 50001 bytes x 100 encode
// 174 -> 77.
constexpr int kWordsU = 4;
constexpr uint32_t kTileU = kApplyThreads * 4 * kWordsU;
static_assert(kTileU == kWordTile, "classic_rules.hpp counts tiles");

// Words of a thread's columns from p on (word v at p + v * kApplyThreads * 4),
// zero where !on.  Both aligned words are read even when one would do: without
// the branch all loads are in flight together, and columns 4 .. 4 + 4 * n keep
// both inside the shard.
__device__ __forceinline__ void ldg_words(const uint8_t *p, const bool *on, uint32_t *x) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  const uint32_t *w = reinterpret_cast<const uint32_t *>(at & ~uintptr_t(3));
  const uint32_t sh = 8 * uint32_t(at & 3);
  uint32_t lo[kWordsU], hi[kWordsU];
#pragma unroll
  for (int v = 0; v < kWordsU; ++v) {
    lo[v] = on[v] ? __ldg(w + v * kApplyThreads) : 0;
    hi[v] = on[v] ? __ldg(w + v * kApplyThreads + 1) : 0;
  }
#pragma unroll
  for (int v = 0; v < kWordsU; ++v) x[v] = __funnelshift_r(lo[v], hi[v], sh);
}

// Writes (ACC: XORs) the warp's words v at p (this lane's address); `on` lanes
// are a prefix of the warp.
template <bool ACC>
__device__ __forceinline__ void stg_words(uint8_t *p, uint32_t v, bool on, uint32_t lane) {
  const uint32_t sh = uint32_t(reinterpret_cast<uintptr_t>(p) & 3);  // uniform
  const uint32_t prev = __shfl_up_sync(0xffffffffu, v, 1);
  const uint32_t active = __ballot_sync(0xffffffffu, on);
  if (!on) return;
  uint8_t *w = p - sh;
  if (sh == 0 || lane) {
    const uint32_t out = sh ? __funnelshift_l(prev, v, 8 * sh) : v;
    uint32_t *dst = reinterpret_cast<uint32_t *>(w);
    *dst = ACC ? (*dst ^ out) : out;
  } else {
    for (uint32_t b = 0; b < 4 - sh; ++b) p[b] = uint8_t(v >> (8 * b)) ^ (ACC ? p[b] : uint8_t(0));
  }
  if (sh && lane == 31u - __clz(active))
    for (uint32_t b = 4 - sh; b < 4; ++b) p[b] = uint8_t(v >> (8 * b)) ^ (ACC ? p[b] : uint8_t(0));
}

template <int C>
__device__ __forceinline__ void unaligned_mac(uint32_t (*acc)[4], const uint8_t *const *ptr, const uint32_t *tbl,
                                              uint64_t col, const bool *on, uint32_t live, uint32_t lane) {
  Lut<C> lut;
  lut_load<C>(lut, lane, [&](int i, uint32_t w) { return __ldg(tbl + i * kTableWords + w); });
  uint32_t x[C][kWordsU];
#pragma unroll
  for (int i = 0; i < C; ++i) ldg_words(ptr[i] + col, on, x[i]);
#pragma unroll
  for (int v = 0; v < kWordsU; ++v) {
    if (uint32_t(v) >= live) break;  // CTA-uniform
    uint32_t y[C], m[Lut<C>::kMixed];
#pragma unroll
    for (int i = 0; i < C; ++i) y[i] = x[i][v];
    lut_index<C>(y, m);
    lut_mac<C>(lut, y, m, acc[v]);
  }
}

template <bool VERIFY, bool ACC>
__global__ void __launch_bounds__(kApplyThreads + 32, 3) k_apply_unaligned(const __grid_constant__ ApplyArgs a) {
  const JobDesc *const jobs = job_list(a);
  const uint8_t *const *const ptrs = ptr_list(a);
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint64_t words = a.len >= 12 ? (a.len - 8) / 4 : 0;
  const uint32_t tiles_per_job = uint32_t((words * 4 + kTileU - 1) / kTileU) + (words ? 0 : 1);
  const uint32_t total = tiles_per_job * a.n_jobs;
  for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
    const uint32_t job = t / tiles_per_job, tile = t - job * tiles_per_job;
    const JobDesc d = jobs[job];
    if (!(d.mode & kJobUnaligned)) continue;  // CTA-uniform
    const uint8_t *const *ptr = ptrs + d.ptr_off;
    if (tid >= kApplyThreads) {
      // The last warp, beside the others' words: the at most 11 columns before
      // and after them, two threads each, with the job's first tile.
      if (tile) continue;
      const uint64_t head = a.len < 4 ? a.len : 4, rest = a.len - head - 4 * words;
      const uint32_t e = lane >> 1;
      const bool mine = e < head + rest;
      const uint64_t c = e < head ? e : 4 * words + e;
      bool bad = false;
      for (uint32_t g = 0; g * 4 < d.n_out; ++g) {
        uint32_t acc = 0;
        if (mine) {
          const uint32_t *tbl = d.tbl + size_t(g) * d.n_in * kTableWords;
#pragma unroll 4
          for (uint32_t j = lane & 1; j < d.n_in; j += 2) {
            const uint32_t x = ptr[j][c];
            acc ^= __ldg(tbl + j * kTableWords + (x & 15)) ^ __ldg(tbl + j * kTableWords + 16 + (x >> 4));
          }
        }
        acc ^= __shfl_xor_sync(0xffffffffu, acc, 1);
#pragma unroll
        for (uint32_t q = 0; q < 2; ++q) {
          const uint32_t r = 2 * (lane & 1) + q, out = 4 * g + r;
          if (mine && out < d.n_out) {
            const uint8_t b = uint8_t(acc >> (8 * r));
            uint8_t *dst = const_cast<uint8_t *>(ptr[d.n_in + out]) + c;
            if (VERIFY) {
              bad |= *dst != b;
              if (d.mode & kJobStore) const_cast<uint8_t *>(ptr[d.n_in + d.n_out + out])[c] = b;
            } else {
              *dst = ACC ? uint8_t(*dst ^ b) : b;
            }
          }
        }
      }
      if (VERIFY && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags + d.flag_idx, 1u);
      continue;
    }
    if (!words) continue;
    const uint64_t word = uint64_t(tile) * (kTileU / 4) + tid, col = 4 + 4 * word;
    const uint64_t left = words - uint64_t(tile) * (kTileU / 4);
    const uint32_t live = uint32_t(left >= kTileU / 4 ? kWordsU : (left + kApplyThreads - 1) / kApplyThreads);
    bool on[kWordsU], bad = false;
#pragma unroll
    for (int v = 0; v < kWordsU; ++v) on[v] = word + v * kApplyThreads < words;
    for (uint32_t g = 0; g * 4 < d.n_out; ++g) {
      uint32_t acc[kWordsU][4];
#pragma unroll
      for (int v = 0; v < kWordsU; ++v)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[v][i] = 0;
      const uint32_t *tbl = d.tbl + size_t(g) * d.n_in * kTableWords;
      uint32_t j = 0;
#pragma unroll 1
      for (; j + 5 <= d.n_in; j += 5) unaligned_mac<5>(acc, ptr + j, tbl + j * kTableWords, col, on, live, lane);
      if (j + 3 <= d.n_in) {
        unaligned_mac<3>(acc, ptr + j, tbl + j * kTableWords, col, on, live, lane);
        j += 3;
      }
#pragma unroll 1
      for (; j < d.n_in; ++j) unaligned_mac<1>(acc, ptr + j, tbl + j * kTableWords, col, on, live, lane);
#pragma unroll
      for (int v = 0; v < kWordsU; ++v) {
        uint32_t o[4];
        transpose4(acc[v], o);
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[v][r] = o[r];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t out = 4 * g + r;
        if (out >= d.n_out) break;  // CTA-uniform
        uint8_t *dst = const_cast<uint8_t *>(ptr[d.n_in + out]) + col;
        if (VERIFY) {
          uint32_t have[kWordsU];
          ldg_words(dst, on, have);
#pragma unroll
          for (int v = 0; v < kWordsU; ++v) bad |= on[v] && have[v] != acc[v][r];
          if (!(d.mode & kJobStore)) continue;
          dst = const_cast<uint8_t *>(ptr[d.n_in + d.n_out + out]) + col;
        }
#pragma unroll
        for (int v = 0; v < kWordsU; ++v) stg_words<ACC>(dst + v * kApplyThreads * 4, acc[v][r], on[v], lane);
      }
    }
    if (VERIFY && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags + d.flag_idx, 1u);
  }
}

// ------------------------------------------------------------------ K3
// GF(2^8) arithmetic from log/exp tables staged in shared memory.
struct SmemGf {
  uint8_t log[256];
  uint8_t exp[512];
  __device__ uint8_t mul(uint8_t a, uint8_t b) const {
    return (a && b) ? exp[log[a] + log[b]] : 0;
  }
  __device__ uint8_t inv(uint8_t a) const { return a ? exp[255 - log[a]] : 0; }
};

__global__ void __launch_bounds__(256) k_decode_tables(DecodeTableArgs a) {
  extern __shared__ uint8_t smem[];
  __shared__ SmemGf gf;
  __shared__ uint8_t factor[256];
  __shared__ int pivot_row;
  __shared__ int singular;
  const DecodeTask task = a.tasks[blockIdx.x];
  const int k = a.k;
  const int w = 2 * k;
  uint8_t *aug = smem;              // k x 2k  [S | I]
  uint8_t *rows = smem + k * w;     // n_out x k composed rows
  for (int i = threadIdx.x; i < 256; i += blockDim.x) gf.log[i] = a.gf_log[i];
  for (int i = threadIdx.x; i < 512; i += blockDim.x) gf.exp[i] = a.gf_exp[i % 255];
  for (int i = threadIdx.x; i < k * w; i += blockDim.x) {
    const int r = i / w, c = i % w;
    uint8_t v;
    if (c < k)
      v = a.matrix[task.survivors[r] * k + c];
    else
      v = (c - k == r) ? 1 : 0;
    aug[i] = v;
  }
  if (threadIdx.x == 0) singular = 0;
  __syncthreads();
  if (task.needs_inverse) {
    for (int col = 0; col < k; ++col) {
      if (threadIdx.x == 0) {
        int p = col;
        while (p < k && aug[p * w + col] == 0) ++p;
        pivot_row = p;
        if (p == k) singular = 1;
      }
      __syncthreads();
      if (singular) break;
      const int p = pivot_row;
      if (p != col)
        for (int c = threadIdx.x; c < w; c += blockDim.x) {
          uint8_t t = aug[p * w + c];
          aug[p * w + c] = aug[col * w + c];
          aug[col * w + c] = t;
        }
      __syncthreads();
      const uint8_t s = gf.inv(aug[col * w + col]);
      __syncthreads();
      for (int c = threadIdx.x; c < w; c += blockDim.x) aug[col * w + c] = gf.mul(s, aug[col * w + c]);
      __syncthreads();
      for (int r = threadIdx.x; r < k; r += blockDim.x) factor[r] = (r == col) ? 0 : aug[r * w + col];
      __syncthreads();
      for (int i = threadIdx.x; i < k * w; i += blockDim.x) {
        const int r = i / w, c = i % w;
        const uint8_t f = factor[r];
        if (f) aug[i] ^= gf.mul(f, aug[col * w + c]);
      }
      __syncthreads();
    }
  }
  if (singular) {
    if (threadIdx.x == 0) a.status[blockIdx.x] = 1;
    return;
  }
  // Compose the requested rows over the survivor columns.  Without missing
  // data the survivors are the data shards in order and the inverse is the
  // identity.
  const int n_out = task.n_out;
  for (int i = threadIdx.x; i < n_out * k; i += blockDim.x) {
    const int t = i / k, c = i % k;
    const int idx = task.targets[t];
    uint8_t v = 0;
    if (idx < k) {
      v = task.needs_inverse ? aug[idx * w + k + c] : uint8_t(task.survivors[c] == idx);
    } else {
      const uint8_t *erow = a.matrix + idx * k;
      if (task.needs_inverse) {
        for (int j = 0; j < k; ++j) v ^= gf.mul(erow[j], aug[j * w + k + c]);
      } else {
        v = erow[task.survivors[c]];
      }
    }
    rows[i] = v;
  }
  __syncthreads();
  // Pack the lookup tables (layout of common.hpp).
  uint32_t *out = task.tbl_out;
  const int groups = (n_out + 3) / 4;
  for (int i = threadIdx.x; i < groups * k * kTableWords; i += blockDim.x) {
    const int e = i % kTableWords, j = (i / kTableWords) % k, g = (i / kTableWords) / k;
    uint32_t word = 0;
    const uint8_t x = e < 16 ? uint8_t(e) : e < 32 ? uint8_t((e - 16) << 4) : uint8_t(e - 32);
    for (int r = 0; r < 4; ++r) {
      const int o = g * 4 + r;
      if (o < n_out) word |= uint32_t(gf.mul(rows[o * k + j], x)) << (8 * r);
    }
    out[i] = word;
  }
  if (threadIdx.x == 0) a.status[blockIdx.x] = 0;
}

// Pair kernel: blockIdx.y selects the pair, the x dimension strides over
// its 16-byte chunks; pairs whose pointers are not both 16-byte aligned, and
// the bytes past the last full chunk, go byte by byte.
template <int MODE>
__global__ void __launch_bounds__(256) k_pairs(const PairOp *pairs, uint32_t *flag) {
  const PairOp p = pairs[blockIdx.y];
  const bool aligned = ((reinterpret_cast<uintptr_t>(p.a) | reinterpret_cast<uintptr_t>(p.b)) & 15) == 0;
  const uint64_t vec = aligned ? p.len / 16 : 0;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  bool bad = false;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < vec; i += stride) {
    const uint4 x = ld_stream(p.a + 16 * i);
    if (MODE == PAIR_COMPARE) {
      const uint4 y = ld_stream(p.b + 16 * i);
      bad |= (x.x != y.x) | (x.y != y.y) | (x.z != y.z) | (x.w != y.w);
    } else {
      uint4 *dst = reinterpret_cast<uint4 *>(p.b + 16 * i);
      const uint4 y = *dst;
      st_stream(p.b + 16 * i, make_uint4(x.x ^ y.x, x.y ^ y.y, x.z ^ y.z, x.w ^ y.w));
    }
  }
  for (uint64_t i = 16 * vec + blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < p.len; i += stride) {
    if (MODE == PAIR_COMPARE)
      bad |= p.a[i] != p.b[i];
    else
      p.b[i] ^= p.a[i];
  }
  if (MODE == PAIR_COMPARE && __any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1u);
}

__global__ void __launch_bounds__(256) k_gather_tables(const uint32_t *full, uint32_t *out, GatherCols cols,
                                                       uint32_t groups, uint32_t k_full, uint32_t n_sel) {
  const uint32_t n = groups * n_sel * kTableWords;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t e = i % kTableWords, j = (i / kTableWords) % n_sel, g = i / (kTableWords * n_sel);
    out[i] = full[(g * k_full + cols.cols[j]) * kTableWords + e];
  }
}

int grid_for(const void *fn, int threads, size_t smem) {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  if (per_sm < 1) per_sm = 1;
  return sms * per_sm;
}

template <int NG, bool VERIFY, bool ACC, int MINB>
void launch_vec(const ApplyArgs &a, cudaStream_t s) {
  static int grid_max = 0;
  const void *fn = (const void *)k_apply_vec<NG, VERIFY, ACC, MINB>;
  if (!grid_max) grid_max = grid_for(fn, kApplyThreads, 0);
  const uint64_t tile = uint64_t(kApplyThreads) * kApplyVec;
  const uint64_t tiles = ((a.len + tile - 1) / tile) * a.n_jobs;
  const int grid = int(tiles < uint64_t(grid_max) ? tiles : grid_max);
  k_apply_vec<NG, VERIFY, ACC, MINB><<<grid, kApplyThreads, 0, s>>>(a);
}

template <int V, int S, bool VERIFY>
void launch_tma(const ApplyArgs &a, cudaStream_t s) {
  constexpr size_t smem = size_t(S) * 4 * kApplyThreads * kApplyVec * V;
  static int grid_max = 0;
  const void *fn = (const void *)k_apply_tma<V, S, VERIFY>;
  ensure_smem_limit(fn, smem);  // per device, set once
  if (!grid_max) grid_max = grid_for(fn, kApplyThreads + 32, smem);
  const uint64_t tile = uint64_t(kApplyThreads) * kApplyVec * V;
  const uint64_t tiles = ((a.len + tile - 1) / tile) * a.n_jobs;
  const int grid = int(tiles < uint64_t(grid_max) ? tiles : grid_max);
  k_apply_tma<V, S, VERIFY><<<grid, kApplyThreads + 32, smem, s>>>(a);
}

template <int K, bool VERIFY>
void launch_reg(const ApplyArgs &a, cudaStream_t s) {
  using Shape = RegShape<K, VERIFY>;
  static int grid_max = 0;
  const void *fn = (const void *)k_apply_reg<K, VERIFY>;
  ensure_smem_limit(fn, Shape::kSmem + 512);  // with the static part it may pass 48 KiB
  if (!grid_max) grid_max = grid_for(fn, kApplyThreads + 32, Shape::kSmem);
  const uint64_t tiles = ((a.len + Shape::kTile - 1) / Shape::kTile) * a.n_jobs;
  const int grid = int(tiles < uint64_t(grid_max) ? tiles : grid_max);
  k_apply_reg<K, VERIFY><<<grid, kApplyThreads + 32, Shape::kSmem, s>>>(a);
}
template <bool VERIFY>
void launch_reg_k(const ApplyArgs &a, cudaStream_t s) {
  switch (a.uni_in) {
#define RS_REG_CASE(K) \
  case K: launch_reg<K, VERIFY>(a, s); break;
    RS_REG_CASE(1) RS_REG_CASE(2) RS_REG_CASE(3) RS_REG_CASE(4) RS_REG_CASE(5) RS_REG_CASE(6) RS_REG_CASE(7)
    RS_REG_CASE(8) RS_REG_CASE(9) RS_REG_CASE(10) RS_REG_CASE(11) RS_REG_CASE(12) RS_REG_CASE(13) RS_REG_CASE(14)
    RS_REG_CASE(15) RS_REG_CASE(16) RS_REG_CASE(17) RS_REG_CASE(18) RS_REG_CASE(19) RS_REG_CASE(20)
#undef RS_REG_CASE
    default: break;
  }
}

template <bool VERIFY, bool ACC>
void launch_unaligned(const ApplyArgs &a, cudaStream_t s) {
  static int grid_max = 0;
  if (!grid_max) grid_max = grid_for((const void *)k_apply_unaligned<VERIFY, ACC>, kApplyThreads + 32, 0);
  const uint64_t tiles = (a.len + kTileU - 1) / kTileU * a.n_jobs;
  const int grid = int(tiles < uint64_t(grid_max) ? tiles : grid_max);
  k_apply_unaligned<VERIFY, ACC><<<grid, kApplyThreads + 32, 0, s>>>(a);
}

// More than 4 outputs: the register-path tile, 8 outputs a pass at 128
// registers (80 registers, three CTAs an SM, spill: 50+20 256 KiB x 32 807
// against 1111 GB/s; one group a pass at 64 registers 1011, three 1066; with
// 4+4 and 5+3 lookups an input, before the shared ones, 672).  At most 4:
// tables in registers up to kRegInputs inputs a job (beyond, they no longer
// fit), the staged tile with tables read per step for wider jobs and for
// launches whose jobs differ in width.  One B200, GB/s, staged tile / tables
// in registers:
//   encode 10+4   1 MiB x 512 4498 / 5351, 64 KiB x 256 3544 / 4374, 8 KiB x 1024 2890 / 3731
//   encode 4+2    1 MiB x 512 4476 / 5345;  16+4 1 MiB x 256 4209 / 4807
//   encode 8+4    4 KiB x 4096 2175 / 4278
//   rebuild 16+4  1 MiB x 256 4109 / 4604;  6+3 256 KiB x 512 4102 / 4765
//   verify 20+4   1 MiB x 128 4036 / 4231;  of one or two inputs: classic_rules.hpp
template <bool VERIFY>
void launch_write_or_verify(const ApplyArgs &a, int variant, cudaStream_t s) {
  if (a.max_out > 4)
    launch_vec<2, VERIFY, false, 2>(a, s);
  else if (variant == 1)
    launch_vec<1, VERIFY, false, 4>(a, s);
  else if (variant == 0 && a.uni_in >= 1 && a.uni_in <= kRegInputs &&
           !(VERIFY && verify_staged(a.uni_in, a.len, a.n_jobs)))
    launch_reg_k<VERIFY>(a, s);
  else
    launch_tma<2, 3, VERIFY>(a, s);
}

}  // namespace

int &apply_variant() {
  static int v = [] {
    const char *e = getenv("RSGPU_APPLY_VARIANT");
    return e ? atoi(e) : 0;
  }();
  return v;
}

cudaError_t launch_apply(const ApplyArgs &a, bool verify, uint64_t max_tail, cudaStream_t s) {
  if (a.n_jobs == 0) return cudaSuccess;
  uint64_t launches = 0;
  if (a.any_vec && a.len >= 16) {
    if (a.accumulate)
      launch_vec<1, false, true, 4>(a, s);
    else if (verify)
      launch_write_or_verify<true>(a, apply_variant(), s);
    else
      launch_write_or_verify<false>(a, apply_variant(), s);
    ++launches;
  }
  if (a.any_unaligned) {
    if (a.accumulate)
      launch_unaligned<false, true>(a, s);
    else if (verify)
      launch_unaligned<true, false>(a, s);
    else
      launch_unaligned<false, false>(a, s);
    ++launches;
  }
  if (max_tail) {
    const uint64_t n = max_tail * a.n_jobs;
    const int threads = 256;
    const uint64_t want = (n + threads - 1) / threads;
    const uint64_t cap = uint64_t(device_sm_count()) * 16;
    const int grid = int(want < cap ? want : cap);
    auto *fn = a.jobs ? (a.accumulate ? k_apply_tail<false, true, false> : verify ? k_apply_tail<true, false, false>
                                                                                 : k_apply_tail<false, false, false>)
                      : (a.accumulate ? k_apply_tail<false, true, true> : verify ? k_apply_tail<true, false, true>
                                                                                : k_apply_tail<false, false, true>);
    fn<<<grid, threads, 0, s>>>(a, max_tail);
    ++launches;
  }
  launch_counter_add(launches);
  return cudaGetLastError();
}

cudaError_t launch_pairs(const PairOp *pairs, uint32_t n, uint64_t max_len, int mode, uint32_t *flag,
                         cudaStream_t s) {
  if (n == 0 || max_len == 0) return cudaSuccess;
  if (n > 65535) return cudaErrorInvalidValue;  // one grid row per pair
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  // About 8 CTAs per SM in total, at least one per 64 KiB of the longest pair.
  const uint64_t per_pair = (max_len + 65535) / 65536;
  uint64_t want = (uint64_t(sms) * 8 + n - 1) / n;
  if (want > per_pair) want = per_pair;
  if (want < 1) want = 1;
  const dim3 grid(uint32_t(want), n);
  if (mode == PAIR_COMPARE)
    k_pairs<PAIR_COMPARE><<<grid, 256, 0, s>>>(pairs, flag);
  else
    k_pairs<PAIR_XOR><<<grid, 256, 0, s>>>(pairs, flag);
  launch_counter_add(1);
  return cudaGetLastError();
}

cudaError_t launch_gather_tables(const uint32_t *full, uint32_t *out, const GatherCols &cols, uint32_t groups,
                                 uint32_t k_full, uint32_t n_sel, cudaStream_t s) {
  const uint32_t n = groups * n_sel * kTableWords;
  if (n == 0) return cudaSuccess;
  const uint32_t grid = (n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184;
  k_gather_tables<<<grid, 256, 0, s>>>(full, out, cols, groups, k_full, n_sel);
  launch_counter_add(1);
  return cudaGetLastError();
}

cudaError_t launch_decode_tables(const DecodeTableArgs &a, int n_tasks, int max_out, cudaStream_t s) {
  if (n_tasks == 0) return cudaSuccess;
  const size_t smem = size_t(a.k) * 2 * a.k + size_t(max_out) * a.k;
  cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(k_decode_tables), smem);
  if (e != cudaSuccess) return e;
  k_decode_tables<<<n_tasks, 256, smem, s>>>(a);
  launch_counter_add(1);
  return cudaGetLastError();
}

}  // namespace rsgpu
