// Raw lane sums of up to kEqBlocks consecutive blocks against the equality
// weights (project_lanes_from_fn, packed_batch.rs:25-41) on the tensor cores:
//   raw[b][j * kC + k] += sum_i v(b, kC * i + j) * weights[i].c[k]
//
// It is a contraction over the packed elements i.  An element is 8 bytes of
// weights in each block (F65521: 8 lanes of s8, KoalaBear: 4 lanes of s16) and
// 16 bytes of table (u8 limbs).  tcgen05.mma kind::i8 reads operands that are
// contracted along their rows in units of 16 bytes, so a row is a pair of
// elements: A's rows are 16 bytes of each of eight blocks (M = 128), in shared
// memory as they lie in HBM (bulk copies); B's are the pair's table entries
// (N = 32), even and odd ones apart (16-byte copies).  The products of an even
// element's lanes with the odd element's limbs and the reverse are dropped.
// KoalaBear's payload bytes are low (unsigned) and high (signed) ones: the MMA
// runs once with A read as signed and once as unsigned, and each lane takes the
// sums that its byte needs.  Sums of kEtGroup pairs stay below
// 2^14 * 255 * 255 < 2^30; the table is read once for all blocks.
//
// The CUDA-core kernels spend their time on multiply-adds (F65521 dp4a with
// byte transposes, KoalaBear widening multiply-adds).  Measured on B200:
//   F65521, eight blocks of 2^27 elements: 1.77 ms, 6.1 TB/s, bound by HBM (4.44
//   on the CUDA cores);
//   KoalaBear, eight blocks of 2^24: 0.236 ms (0.813), of 2^28: 3.53 ms, 6.1
//   TB/s, bound by HBM; three blocks of 2^28: 2.86 ms (6.28), 3.7 TB/s, bound by
//   the 16 MMAs of a stage, which take eight blocks' rows either way.
// Neighbouring CTAs take neighbouring stages: a contiguous run of stages per CTA
// put 1300 streams on distant pages (F65521 3.85 against 3.35 ms, before one lane
// per block issued the copies).  Chunks 4096 bytes apart put a row's 16-byte
// units on the same banks; 16 bytes more per chunk brought three KoalaBear blocks
// of 2^28 from 3.30 to 2.86 ms.
#pragma once
#include <cstdint>

#include "../device/tcgen05.cuh"
#include "commit.cuh"
#include "open.cuh"

namespace QFD_NS {

constexpr int kEtEpiWarps = 4, kEtTableWarps = 2, kEtThreads = 32 * (kEtEpiWarps + 2 + kEtTableWarps);
constexpr uint32_t kEtPairs = 256;                  // pairs (rows) of a stage
constexpr uint32_t kEtChunkBytes = 16 * kEtPairs;   // of one block, or of one half of the table
constexpr uint32_t kEtPitch = kEtChunkBytes + 16;   // of chunks in shared memory: a row's 16-byte units on different banks
constexpr uint32_t kEtStageBytes = (kEqBlocks + 2) * kEtPitch;
constexpr int kEtStages = 5;
constexpr uint32_t kEtGroup = 64;                   // stages per read of the sums
constexpr size_t kEtSmem = size_t(kEtStages) * kEtStageBytes + 1024 + 256;
constexpr bool kEtBytes = sizeof(Wt) == 2;          // payloads are a low and a high byte
constexpr uint32_t kEtCols = kEtBytes ? 64 : 32;    // TMEM columns of one buffer

// The part of a chunk at `to` that the bulk copy does not bring: from the last
// whole 16 bytes of the `avail` that exist on, zero past them.  One warp.
__device__ __forceinline__ void et_zero_tail(unsigned char* to, const unsigned char* src, uint32_t avail, int lane) {
  const uint32_t whole = avail & ~15u;
  for (uint32_t u = whole / 16 + lane; u < kEtPairs; u += 32) {
    uint32_t w[4] = {0, 0, 0, 0};
    if (16 * u < avail)
      for (uint32_t j = 0; j < avail - whole; ++j) w[j >> 2] |= uint32_t(src[whole + j]) << (8 * (j & 3));
    reinterpret_cast<uint4*>(to)[u] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// bva is 16-byte aligned and m a multiple of 2 * kEtPairs (the launcher checks
// both).  n_stages = m / 512.
__global__ void __launch_bounds__(kEtThreads, 1) k_eq_project_tc(const Wt* __restrict__ bva, uint64_t active, uint64_t block_len,
                                                                 uint64_t first_block, int nb, uint32_t n_stages,
                                                                 const Fe* __restrict__ weights, unsigned long long* __restrict__ raw,
                                                                 int* error) {
  extern __shared__ unsigned char et_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(et_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* tail = base + kEtStages * kEtStageBytes;
  const uint32_t bars = tc5::smem_addr(tail);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto landed = [&](int s) { return bars + 8 * s; };                    // copies -> MMA
  auto unused = [&](int s) { return bars + 8 * (kEtStages + s); };      // MMA -> copies
  auto full = [&](int b) { return bars + 8 * (2 * kEtStages + b); };    // MMA -> epilogue: sums of a group
  auto empty = [&](int b) { return bars + 8 * (2 * kEtStages + 2 + b); };
  const uint32_t tmem_slot = bars + 8 * (2 * kEtStages + 4);
  bool lost = false;
  auto wait = [&](uint32_t bar, uint32_t parity) {
    if (tc5::mbar_try(bar, parity & 1)) return;
    if (!lost && !tc5::mbar_wait(bar, parity & 1)) {
      lost = true;
      *error = 1;
    }
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kEtStages; ++s) {
      tc5::mbar_init(landed(s), 1 + 32 * kEtTableWarps);
      tc5::mbar_init(unused(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc5::mbar_init(full(b), 1);
      tc5::mbar_init(empty(b), kEtEpiWarps);
    }
  }
  if (warp == kEtEpiWarps + 1) tc5::tmem_alloc(tmem_slot, 2 * kEtCols);
  tc5::fence_async_smem();
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tail + 8 * (2 * kEtStages + 4));
  // Neighbouring CTAs take neighbouring stages.
  const uint32_t n_own = blockIdx.x < n_stages ? (n_stages - blockIdx.x - 1) / gridDim.x + 1 : 0;
  const uint32_t n_groups = (n_own + kEtGroup - 1) / kEtGroup;

  if (warp < kEtEpiWarps) {
    // Thread m: byte m & 15 of the pair in block m >> 4.
    const uint32_t b = threadIdx.x >> 4, y = threadIdx.x & 15;
    const bool odd = y >= 8;
    long long tot[kC];
#pragma unroll
    for (int k = 0; k < kC; ++k) tot[k] = 0;
    for (uint32_t n = 0; n < n_groups; ++n) {
      wait(full(n & 1), n >> 1);
      tc5::fence_after_sync();
      uint32_t d[32], s[16];
      tc5::tmem_ld32(d, tmem + kEtCols * (n & 1) + (uint32_t(warp) << 21));
#pragma unroll
      for (int i = 0; i < 16; ++i) s[i] = odd ? d[16 + i] : d[i];
      if constexpr (kEtBytes) {
        tc5::tmem_ld32(d, tmem + kEtCols * (n & 1) + 32 + (uint32_t(warp) << 21));
        if (!(y & 1))
#pragma unroll
          for (int i = 0; i < 16; ++i) s[i] = odd ? d[16 + i] : d[i];
      }
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(empty(n & 1));
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        constexpr int kLimbs = 16 / kC;
        long long x = 0;
#pragma unroll
        for (int q = kLimbs - 1; q >= 0; --q) x = x * 256 + int32_t(s[kLimbs * k + q]);
        if constexpr (kEtBytes) tot[k] += (long long)mod_i64(x) << (8 * (y & 1));  // residues: a group's sum is below 2^55
        else tot[k] += x;
      }
    }
    if (int(b) < nb) {
      unsigned long long* to = raw + uint64_t(b) * kEqRaw + (kEtBytes ? (y & 7) >> 1 : y & 7) * kC;
#pragma unroll
      for (int k = 0; k < kC; ++k) atomicAdd(to + k, (unsigned long long)(kEtBytes ? (long long)mod_i64(tot[k]) : tot[k]));
    }
  } else if (warp == kEtEpiWarps) {
    // The blocks' weights, a lane per block.
    const unsigned char* src = reinterpret_cast<const unsigned char*>(bva);
    const uint64_t end = active * sizeof(Wt);
    const uint64_t at0 = (first_block + lane) * block_len * sizeof(Wt);
    for (uint32_t st = blockIdx.x, n = 0; n < n_own; st += gridDim.x, ++n) {
      const int s = n % kEtStages;
      unsigned char* stage = base + s * kEtStageBytes;
      if (n >= kEtStages) wait(unused(s), n / kEtStages - 1);
      const uint64_t at = at0 + uint64_t(st) * kEtChunkBytes;
      const uint32_t avail = lane >= nb || at >= end ? 0u : uint32_t(end - at < kEtChunkBytes ? end - at : kEtChunkBytes);
      const uint32_t bytes = avail & ~15u;
      uint32_t ragged = __ballot_sync(0xffffffffu, lane < nb && avail < kEtChunkBytes);
      uint32_t total = uint32_t(nb) * kEtChunkBytes;
      if (ragged) {
        total = __reduce_add_sync(0xffffffffu, bytes);
        for (; ragged; ragged &= ragged - 1) {
          const int b = __ffs(ragged) - 1;
          et_zero_tail(stage + b * kEtPitch, src + __shfl_sync(0xffffffffu, at, b), __shfl_sync(0xffffffffu, avail, b), lane);
        }
        tc5::fence_async_smem();
      }
      __syncwarp();
      if (lane == 0) tc5::mbar_expect(landed(s), total);
      __syncwarp();
      if (bytes) tc5::bulk_load(tc5::smem_addr(stage) + lane * kEtPitch, src + at, bytes, landed(s));
    }
    // No copy is in flight when the CTA ends, also after a wait that gave up.
    for (uint32_t i = n_own < kEtStages ? 0 : n_own - kEtStages; i < n_own; ++i) tc5::mbar_wait(landed(i % kEtStages), i / kEtStages & 1);
  } else if (warp > kEtEpiWarps + 1) {
    // The table: lanes take consecutive elements, even ones to the first half.
    const uint32_t t = uint32_t(warp - kEtEpiWarps - 2) * 32 + lane;
    for (uint32_t st = blockIdx.x, n = 0; n < n_own; st += gridDim.x, ++n) {
      const int s = n % kEtStages;
      unsigned char* to = base + s * kEtStageBytes + kEqBlocks * kEtPitch + (lane & 1) * kEtPitch + (t >> 1) * 16;
      if (n >= kEtStages) wait(unused(s), n / kEtStages - 1);
      const Fe* w = weights + uint64_t(st) * (2 * kEtPairs) + t;
#pragma unroll
      for (int i = 0; i < int(2 * kEtPairs / (32 * kEtTableWarps)); ++i)
        cp_async16(to + 256 * kEtTableWarps * i, w + 32 * kEtTableWarps * i);
      tc5::mbar_arrive_copies(landed(s));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (lane == 0) {
    constexpr uint32_t kIdesc = tc5::idesc_i8(128, 32) | (1u << 15);  // both operands contracted along their rows
    constexpr uint32_t kUnsigned = kIdesc & ~(1u << 7);               // A as u8
    for (uint32_t n = 0; n < n_own; ++n) {
      const int s = n % kEtStages;
      const uint32_t g = n / kEtGroup, d = tmem + kEtCols * (g & 1);
      if (n % kEtGroup == 0 && g >= 2) wait(empty(g & 1), (g >> 1) - 1);
      wait(landed(s), n / kEtStages);
      tc5::fence_async_smem();  // the table's copies and the zeros
      tc5::fence_after_sync();
      const uint32_t a = tc5::smem_addr(base) + s * kEtStageBytes, b = a + kEqBlocks * kEtPitch;
#pragma unroll
      for (uint32_t j = 0; j < kEtPairs / 32; ++j) {
        const uint64_t da = tc5::smem_desc(a + 512 * j, 128, kEtPitch, 0), db = tc5::smem_desc(b + 512 * j, 128, kEtPitch, 0);
        const uint32_t more = n % kEtGroup + j > 0;
        tc5::mma_i8(d, da, db, kIdesc, more);
        if constexpr (kEtBytes) tc5::mma_i8(d + 32, da, db, kUnsigned, more);
      }
      tc5::mma_commit(unused(s));
      if (n % kEtGroup == kEtGroup - 1 || n + 1 == n_own) tc5::mma_commit(full(g & 1));
    }
    // No MMA is in flight and no arrival on its way when the CTA ends, also
    // after a wait that gave up.
    for (uint32_t i = n_own < kEtStages ? 0 : n_own - kEtStages; i < n_own; ++i) tc5::mbar_wait(unused(i % kEtStages), i / kEtStages & 1);
    for (uint32_t g = n_groups < 2 ? 0 : n_groups - 2; g < n_groups; ++g) tc5::mbar_wait(full(g & 1), g >> 1 & 1);
  }
  __syncwarp();
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == kEtEpiWarps + 1) tc5::tmem_free(tmem, 2 * kEtCols);
}

}  // namespace QFD_NS
