// TBV lane projections of F65521 terms with 16 lanes on the tensor cores
// (tbv.rs:288-352): S[tile][lane] = sum over the tile's rows r of
// v[r][lane] * lo[r], times the tile's high weight.
//
// It is a contraction over rows: weights (s8) against the table's storage
// bytes (u8 limbs, 16 columns), exact in s32 for 4096 rows (4096 * 128 * 255 <
// 2^27).  Memory holds both operands as tcgen05.mma kind::i8 reads them without
// swizzle: a row's 16 lanes (or an element's 16 bytes) contiguous, rows 16
// bytes apart.  One MMA takes 32 rows of eight tiles (M = 8 tiles x 16 lanes,
// N = 16), so the weights go from HBM to shared memory by bulk copies and are
// never touched by a CUDA core.  The dp4a kernel spends its time on byte
// transposes and the reduction across threads at each tile's end.
//
// Measured on B200: 872 M weights in 52 terms 0.150 ms, 5.8 TB/s (0.635 ms in the
// dp4a kernel), 8.05 G weights 1.22 ms, 6.6 TB/s: what is left is HBM.  Lists of
// small terms are bound by the latency of a group's loads: 20000 terms of 256
// rows 172 us (305).
#pragma once
#include <cstdint>

#include "../device/tcgen05.cuh"
#include "open.cuh"

namespace QFD_NS {

constexpr int kPmEpiWarps = 4, kPmThreads = 32 * (kPmEpiWarps + 2);
constexpr int kPmTiles = 8;          // tiles per group: M = 128
constexpr uint32_t kPmRows = 256;    // rows of a stage
constexpr uint32_t kPmTileBytes = 16 * kPmRows, kPmStageBytes = (kPmTiles + 1) * kPmTileBytes;
constexpr int kPmStages = 6;
constexpr size_t kPmSmem = size_t(kPmStages) * kPmStageBytes + 1024 + 256;

// Group `g`: up to eight tiles of one list entry; the term's last tile, when
// it has fewer rows than the others, is a group of its own.
__host__ __device__ inline bool pm_ragged(const TermTiles& T) {
  return ((uint64_t(T.tile_skip) + T.tiles) << T.lb) > T.rows;
}
__host__ __device__ inline uint32_t pm_groups(const TermTiles& T) {
  const uint32_t full = T.tiles - (pm_ragged(T) ? 1 : 0);
  return (full + kPmTiles - 1) / kPmTiles + (pm_ragged(T) ? 1 : 0);
}
// Stages of a group of tiles of `rows` rows.
__host__ __device__ inline uint32_t pm_stages(uint64_t rows) { return uint32_t((rows + kPmRows - 1) / kPmRows); }
struct PmGroup {
  TermTiles T;
  uint32_t first, tiles;  // tiles of the entry
  uint32_t rows;          // of each
};
__device__ __forceinline__ PmGroup pm_group(const TermTiles* __restrict__ terms, int n_terms, int& ti, uint32_t g) {
  while (ti + 1 < n_terms && terms[ti + 1].first_group <= g) ++ti;
  PmGroup G;
  G.T = terms[ti];
  const uint32_t full = G.T.tiles - (pm_ragged(G.T) ? 1 : 0), j = g - G.T.first_group, whole = (full + kPmTiles - 1) / kPmTiles;
  G.first = j < whole ? j * kPmTiles : full;
  G.tiles = j < whole ? min(full - G.first, uint32_t(kPmTiles)) : 1u;
  G.rows = j < whole ? 1u << G.T.lb : uint32_t(G.T.rows & ((uint64_t(1) << G.T.lb) - 1));
  return G;
}

// A run of the groups per CTA (list.first).  Every row of every entry lies below the end of the weights, and the weights and offsets are 16-byte
// aligned (the launcher checks both).
__global__ void __launch_bounds__(kPmThreads, 1) k_project_terms_mma(const int8_t* __restrict__ bva, const TermTiles* __restrict__ terms,
                                                                     int n_terms, const __grid_constant__ TermGroups list,
                                                                     const Fe* __restrict__ tables, Fe* __restrict__ out, int* error) {
  extern __shared__ unsigned char pm_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pm_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* tail = base + kPmStages * kPmStageBytes;
  const uint32_t bars = tc5::smem_addr(tail);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto landed = [&](int s) { return bars + 8 * s; };                    // copies -> MMA
  auto unused = [&](int s) { return bars + 8 * (kPmStages + s); };      // MMA -> copies
  auto full = [&](int b) { return bars + 8 * (2 * kPmStages + b); };    // MMA -> epilogue: sums of a group
  auto empty = [&](int b) { return bars + 8 * (2 * kPmStages + 2 + b); };
  const uint32_t tmem_slot = bars + 8 * (2 * kPmStages + 4);
  bool lost = false;
  auto wait = [&](uint32_t bar, uint32_t parity) {
    if (tc5::mbar_try(bar, parity & 1)) return;
    if (!lost && !tc5::mbar_wait(bar, parity & 1)) {
      lost = true;
      *error = 1;
    }
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPmStages; ++s) {
      tc5::mbar_init(landed(s), 1);
      tc5::mbar_init(unused(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc5::mbar_init(full(b), 1);
      tc5::mbar_init(empty(b), kPmEpiWarps);
    }
  }
  if (warp == kPmEpiWarps + 1) tc5::tmem_alloc(tmem_slot, 32);
  tc5::fence_async_smem();
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tail + 8 * (2 * kPmStages + 4));
  const uint32_t g0 = list.first[blockIdx.x], g1 = list.first[blockIdx.x + 1];
  int ti = 0;
  for (int last = n_terms - 1; ti < last;) {  // the entry of group g0
    const int mid = (ti + last + 1) >> 1;
    if (terms[mid].first_group <= g0) ti = mid;
    else last = mid - 1;
  }

  if (warp < kPmEpiWarps) {
    // Thread m: lane m & 15 of the group's tile m >> 4.
    const uint32_t m = threadIdx.x;
    for (uint32_t g = g0, n = 0; g < g1; ++g, ++n) {
      const PmGroup G = pm_group(terms, n_terms, ti, g);
      wait(full(n & 1), n >> 1);
      tc5::fence_after_sync();
      uint32_t s[16];
      tc5::tmem_ld16(s, tmem + 16 * (n & 1) + (uint32_t(warp) << 21));
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(empty(n & 1));
      if ((m >> 4) < G.tiles) {
        const uint32_t k = G.first + (m >> 4);  // tile of this list entry
        Fr v;
#pragma unroll
        for (int c = 0; c < kC; ++c) v.c[c] = red_signed(int64_t(int32_t(s[2 * c])) + 256 * int64_t(int32_t(s[2 * c + 1])));
        store(out + (size_t(G.T.first_tile) + k) * 16 + (m & 15), mul(tile_high(G.T, tables, uint64_t(k) + G.T.tile_skip), v));
      }
    }
  } else if (warp == kPmEpiWarps) {
    uint32_t n = 0;  // stages so far
    for (uint32_t g = g0; g < g1; ++g) {
      const PmGroup G = pm_group(terms, n_terms, ti, g);
      const int8_t* v = bva + (G.T.offset + ((uint64_t(G.first) + G.T.tile_skip) << G.T.lb) * 16);
      const Fe* w = tables + G.T.lo_off;
      for (uint32_t r = 0; r < G.rows; r += kPmRows, ++n) {
        const int s = n % kPmStages;
        const uint32_t rows = min(kPmRows, G.rows - r);
        unsigned char* stage = base + s * kPmStageBytes;
        if (n >= kPmStages) wait(unused(s), n / kPmStages - 1);
        if (rows & 31) {
          // The table's rows up to the MMA's 32 are zero, so that what the
          // weights' side holds there does not count.
          const uint32_t pad = 32 - (rows & 31);
          if (uint32_t(lane) < pad) reinterpret_cast<uint4*>(stage + kPmTiles * kPmTileBytes)[rows + lane] = make_uint4(0, 0, 0, 0);
          tc5::fence_async_smem();
        }
        __syncwarp();
        if (lane == 0) {
          const uint32_t to = tc5::smem_addr(stage);
          tc5::mbar_expect(landed(s), 16 * rows * (G.tiles + 1));
          for (uint32_t t = 0; t < G.tiles; ++t)
            tc5::bulk_load(to + t * kPmTileBytes, v + ((uint64_t(t) << G.T.lb) + r) * 16, 16 * rows, landed(s));
          tc5::bulk_load(to + kPmTiles * kPmTileBytes, w + r, 16 * rows, landed(s));
        }
      }
    }
    // No copy is in flight when the CTA ends, also after a wait that gave up.
    for (uint32_t i = n < kPmStages ? 0 : n - kPmStages; i < n; ++i) tc5::mbar_wait(landed(i % kPmStages), i / kPmStages & 1);
  } else if (lane == 0) {
    constexpr uint32_t kIdesc = tc5::idesc_i8(128, 16) | (1u << 15);  // both operands contracted along their rows
    uint32_t n = 0;
    for (uint32_t g = g0, k = 0; g < g1; ++g, ++k) {
      const PmGroup G = pm_group(terms, n_terms, ti, g);
      if (k >= 2) wait(empty(k & 1), (k >> 1) - 1);
      tc5::fence_after_sync();
      for (uint32_t r = 0; r < G.rows; r += kPmRows, ++n) {
        const int s = n % kPmStages;
        wait(landed(s), n / kPmStages);
        const uint32_t a = tc5::smem_addr(base) + s * kPmStageBytes, b = a + kPmTiles * kPmTileBytes;
        const uint32_t steps = (min(kPmRows, G.rows - r) + 31) / 32;
        for (uint32_t j = 0; j < steps; ++j)
          tc5::mma_i8(tmem + 16 * (k & 1), tc5::smem_desc(a + 512 * j, 128, kPmTileBytes, 0), tc5::smem_desc(b + 512 * j, 128, 128, 0),
                      kIdesc, r + j > 0);
        tc5::mma_commit(unused(s));
      }
      tc5::mma_commit(full(k & 1));
    }
    // No MMA is in flight and no arrival on its way when the CTA ends, also
    // after a wait that gave up.
    const uint32_t k1 = g1 - g0;
    for (uint32_t i = n < kPmStages ? 0 : n - kPmStages; i < n; ++i) tc5::mbar_wait(unused(i % kPmStages), i / kPmStages & 1);
    for (uint32_t k = k1 < 2 ? 0 : k1 - 2; k < k1; ++k) tc5::mbar_wait(full(k & 1), k >> 1 & 1);
  }
  __syncwarp();
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == kPmEpiWarps + 1) tc5::tmem_free(tmem, 32);
}

}  // namespace QFD_NS
