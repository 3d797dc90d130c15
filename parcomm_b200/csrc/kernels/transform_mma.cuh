// The transform passes of the codeword encoding on the tensor cores.
//
// A pass takes tiles of 8192 packed elements (128 KiB) through up to 26 levels
// of the Mobius transform or of the unnormalised WHT (packed.rs:708-752,
// qafold_short.rs:975-1002), each level a 2 x 2 map on one index bit.  Up to
// seven levels together are one 128 x 128 matrix with entries 0, 1, -1 (a
// Kronecker product of 2 x 2 maps, with identities for the bits of the seven
// that take no level), the same for every coefficient and every other index,
// so they are a contraction: tcgen05.mma kind::i8 multiplies it with the
// elements' storage bytes as unsigned limbs.  An element's 16 bytes are 16
// columns of the product; a coefficient is the weighted sum of its limbs'
// columns (exact in s32 per limb), reduced once per stage.  No conversion
// precedes the MMA: the bytes in HBM are the limbs.
//
// Tile element bits are 13 slots.  Stage X contracts slots 0..6; stage Y
// contracts seven slots that share with X slot 0 (kTileCfg: 13 levels over the
// low 13 index bits) or slots 0 and 1 (kStridedCfg: 10 levels over high index
// bits; the shared slots and slot 12 are runs of consecutive elements).  The
// tile lies in shared memory as the MMA's N-major operand B under the 128-byte
// swizzle: 16-byte unit bits [n n n | k k k | k k | n | . . . .], the low
// three XORed with the next three.  A stage works in four chunks of 128 x 256
// products; a chunk occupies the same addresses in the layouts of both stages,
// so its results overwrite it in either one.  Stores, loads and MMA reads are
// free of bank conflicts.
//
// Warps 0..15 run the epilogue (TMEM -> registers -> combine, reduce, pack ->
// shared memory or HBM), warp 16 issues the MMAs, the others load.  TMEM holds
// two chunks of 256 columns, so the MMAs run ahead of the epilogue; K step j of
// a stage needs only chunk j of the stage before.  The last stage is X, whose
// chunks are 32 KiB regions of the tile: shared memory is a ring of five or six
// regions, and a region is loaded anew once the last stage's MMA has read it.
#pragma once
#include <cstdint>

#include "../device/tcgen05.cuh"
#include "commit.cuh"

namespace QFD_NS {

constexpr int kTcEpiWarps = 16;
// Copies need two warps; packing weights is arithmetic and takes four.
constexpr int tc_load_warps(int src) { return src == 1 ? 4 : 2; }
constexpr int tc_threads(int src) { return 32 * (kTcEpiWarps + 1 + tc_load_warps(src)); }
constexpr int kTcTileLog = 13;
constexpr uint32_t kTcRegionBytes = 32768, kTcMatBytes = 16384;  // a tile is four regions
// Regions of the ring: what the matrices leave of 227 KiB.
constexpr int tc_regions(int mats) { return mats > 2 ? 5 : 6; }
// The ring, the matrices, barriers, and the slack of a 1 KiB alignment.
constexpr size_t tc_smem(int mats) { return size_t(tc_regions(mats)) * kTcRegionBytes + size_t(mats) * kTcMatBytes + 1024 + 256; }

struct TcPass {
  const void* src;    // elements, or weights (kTcWeights)
  Fe* dst;            // where the last stage stores
  Fe* mid;            // kMidStore: where the middle values go
  const Fe* alpha;    // kMidAlpha: the row factors
  int* error;         // set when a wait gives up (host-mapped)
  uint64_t active, src_base;  // kTcWeights: entries, and the block's first
  uint32_t stride[kTcTileLog];  // of each slot, in codeword elements
  int logR, lo, k, cb;        // the tile's base index (tc_tile_base)
  uint32_t mask_x, mask_y;    // K bits of a stage that take a level
  uint32_t c256;              // 256, opaque to the compiler: a multiply-add instead of a shift and an add
  int col_log;                // kMidAlpha: log2 of the columns of whole tiles
  uint32_t n_tiles;
};
enum TcMid { kMidNone = 0, kMidStore = 1, kMidAlpha = 2 };
enum TcSrc { kTcElements = 0, kTcWeights = 1, kTcLinear = 2 };  // kTcLinear: elements at their logical index
enum TcConfig { kTileCfg = 0, kStridedCfg = 1 };

// Slots by role: of K bit i, N bit i, chunk bit i, and unit bit of each stage.
template <int CFG, bool X>
struct TcLayout {
  static constexpr int k(int i) {
    constexpr int t[2][7] = {{0, 7, 8, 9, 10, 11, 12}, {0, 1, 7, 8, 9, 10, 11}};
    return X ? i : t[CFG][i];
  }
  static constexpr int n(int i) {
    constexpr int t[2][2][4] = {{{3, 1, 2, 4}, {9, 7, 8, 10}}, {{3, 4, 2, 12}, {8, 9, 7, 12}}};
    return t[CFG][X][i];
  }
  static constexpr int chunk(int i) { return X ? (CFG == kTileCfg ? 11 : 10) + i : 5 + i; }
  // Unit within a region: bits 9, 10 are slots 5, 6.  The region is stage Y's
  // last two K slots.
  static constexpr uint32_t unit(uint32_t e) {
    uint32_t u = 0;
    for (int i = 0; i < 3; ++i) {
      u |= ((e >> n(i) ^ e >> k(i)) & 1u) << i;
      u |= (e >> k(i) & 1u) << (3 + i);
    }
    for (int i = 0; i < 2; ++i) {
      u |= (e >> k(3 + i) & 1u) << (6 + i);
      u |= (e >> (5 + i) & 1u) << (9 + i);
    }
    return u | (e >> n(3) & 1u) << 8;
  }
  // Slots of epilogue lane m (the contracted output index) and of column group
  // n (16 per chunk).
  static constexpr uint32_t of_m(uint32_t m) {
    uint32_t e = 0;
    for (int i = 0; i < 7; ++i) e |= (m >> i & 1u) << k(i);
    return e;
  }
  static constexpr uint32_t of_n(uint32_t v) {
    uint32_t e = 0;
    for (int i = 0; i < 4; ++i) e |= (v >> i & 1u) << n(i);
    return e;
  }
};

// Codeword index of tile `tile`'s element 0: the tile numbers the index bits
// outside [lo, lo + k) and above the cb run bits.
__device__ __forceinline__ uint32_t tc_tile_base(const TcPass& p, uint32_t tile) {
  const uint32_t g = tile << p.cb;
  return msg_addr32(((g >> p.lo) << (p.lo + p.k)) | (g & ((1u << p.lo) - 1u)), p.logR);
}

// Entry (m, k) of the matrix of OP's levels on the index bits of `mask`.
template <int OP>
__device__ __forceinline__ uint32_t tc_entry(uint32_t m, uint32_t k, uint32_t mask) {
  if ((m ^ k) & ~mask) return 0;
  if (OP == kWht) return (__popc(m & k & mask) & 1) ? 0xffu : 1u;
  if (k & ~m) return 0;
  return (__popc(m & ~k) & 1) ? 0xffu : 1u;
}
// The matrix as the K-major operand A: rows of 128 bytes, 128-byte swizzle.
template <int OP>
__device__ __forceinline__ void tc_matrix(unsigned char* dst, uint32_t mask) {
  for (uint32_t u = threadIdx.x; u < kTcMatBytes / 16; u += blockDim.x) {
    const uint32_t m = u >> 3, c = u & 7;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) w[i] |= tc_entry<OP>(m, 16 * c + 4 * i + j, mask) << (8 * j);
    }
    reinterpret_cast<uint4*>(dst)[(m << 3) | (c ^ (m & 7))] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The weights of two consecutive elements (8 bytes each), zero past `active`.
// `wide`: both are there, at a 16-byte boundary.
__device__ __forceinline__ uint4 tc_weights(const TcPass& p, uint64_t element, bool wide) {
  const Wt* bva = static_cast<const Wt*>(p.src);
  const uint64_t g = p.src_base + uint64_t(kC) * element;
  if (wide) return *reinterpret_cast<const uint4*>(bva + g);
  if (g + 2 * kC <= p.active) {
    const uint2 a = *reinterpret_cast<const uint2*>(bva + g), b = *reinterpret_cast<const uint2*>(bva + g + kC);
    return make_uint4(a.x, a.y, b.x, b.y);
  }
  constexpr int kPer = 4 / int(sizeof(Wt));
  constexpr uint32_t kMask = (1u << (8 * sizeof(Wt))) - 1u;
  uint32_t w[4] = {0, 0, 0, 0};
  for (int k = 0; k < 2 * kC; ++k)
    if (g + k < p.active) w[k / kPer] |= (uint32_t(bva[g + k]) & kMask) << (8 * int(sizeof(Wt)) * (k % kPer));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Barriers (8 bytes each, from `bars`).  Every wait is bounded; a wait that
// gives up sets the error flag, and later waits do not wait.
struct TcBars {
  uint32_t bars;
  int* error;
  bool lost;
  __device__ uint32_t full(int b) const { return bars + 8 * b; }           // MMA -> epilogue: TMEM buffer b holds a chunk
  __device__ uint32_t empty(int b) const { return bars + 16 + 8 * b; }     // epilogue -> MMA: buffer b has been read
  __device__ uint32_t written(int c) const { return bars + 32 + 8 * c; }   // epilogue -> MMA: chunk c of a stage is in the tile
  __device__ uint32_t unused(int r) const { return bars + 64 + 8 * r; }    // MMA -> loads: region r may be loaded anew
  __device__ uint32_t loaded(int r) const { return bars + 112 + 8 * r; }   // loads -> MMA: region r is there
  __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity) {
    if (tc5::mbar_try(bar, parity & 1)) return;
    if (!lost && !tc5::mbar_wait(bar, parity & 1)) {
      lost = true;
      *error = 1;
    }
  }
};
// Ring position of a region that advances by four per tile.
template <int NR>
__device__ __forceinline__ uint32_t tc_next(uint32_t r) { return r + 4 >= NR ? r + 4 - NR : r + 4; }

// The epilogue of one chunk: per element the limb sums' reduction and
// fin(i, Fr&) on the canonical value; TO 1 / 2 stores it into `region` in the
// layout of stage X / Y at unit u0 of chunk 0, 0 leaves it to fin.
// PARTS 2 takes the columns in two halves, for fewer registers.
template <int CFG, bool X, int TO, int PARTS, class Before, class Fin>
__device__ __forceinline__ void tc_chunk(TcBars& B, uint32_t region, uint32_t tmem, uint32_t u, int c, uint32_t u0, uint32_t c256,
                                         Before before, Fin fin) {
  using L = TcLayout<CFG, X>;
  using To = TcLayout<CFG, TO == 1>;
  before();
  B.wait(B.full(u & 1), u >> 1);
  tc5::fence_after_sync();
  const uint32_t uc = (X ? u0 : u0 ^ uint32_t(c) << 9) << 4;  // stage Y's chunk bits, alike in both layouts
#pragma unroll
  for (int h = 0; h < PARTS; ++h) {
    uint32_t d[64 / PARTS];
    if constexpr (PARTS == 1) tc5::tmem_ld64(d, tmem + 256u * (u & 1));
    else tc5::tmem_ld32(d, tmem + 256u * (u & 1) + 32u * h);
    if (h == PARTS - 1) {
      tc5::fence_before_sync();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) tc5::mbar_arrive(B.empty(u & 1));
    }
#pragma unroll
    for (int q = 0; q < 4 / PARTS; ++q) {
      const int i = h * (4 / PARTS) + q;
      uint32_t s[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) s[j] = d[16 * q + j];
      Fr v = limb_sums(s, c256);
      fin(i, v);
      if (TO) tc5::store_shared(region + (uc ^ To::unit(L::of_n(i)) << 4), pack_fe(v));
    }
  }
  if (TO) {
    tc5::fence_async_smem();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) tc5::mbar_arrive(B.written(c));
  }
}

// One pass.  Stages: without OP2 Y then X, or X alone when stage Y takes no
// level (HASY false); with OP2 X Y mid Y X, or X mid X.
template <int CFG, int SRC, int OP1, int OP2, int MID, bool HASY>
__global__ void __launch_bounds__(tc_threads(SRC), 1) k_transform(const __grid_constant__ TcPass p) {
  extern __shared__ unsigned char tc_smem_raw[];
  using LX = TcLayout<CFG, true>;
  using LY = TcLayout<CFG, false>;
  constexpr bool kTwo = OP2 >= 0;
  constexpr bool kFirstX = kTwo || !HASY;
  constexpr bool kOther = kTwo && OP1 != OP2;
  constexpr int kParts = SRC == kTcWeights ? 2 : 1;  // 21 warps leave 80 registers
  constexpr int kStages = (HASY ? 2 : 1) * (kTwo ? 2 : 1);
  constexpr int kMats = (HASY ? 2 : 1) * (kOther ? 2 : 1), NR = tc_regions(kMats);
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* mats = ring + NR * kTcRegionBytes;
  unsigned char* tail = mats + kMats * kTcMatBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // Matrices: stage X of OP1, stage Y of OP1, then those of OP2.
  tc_matrix<OP1>(mats, p.mask_x);
  if (HASY) tc_matrix<OP1>(mats + kTcMatBytes, p.mask_y);
  if (kOther) {
    tc_matrix<(OP2 >= 0 ? OP2 : 0)>(mats + (HASY ? 2 : 1) * kTcMatBytes, p.mask_x);
    if (HASY) tc_matrix<(OP2 >= 0 ? OP2 : 0)>(mats + 3 * kTcMatBytes, p.mask_y);
  }
  TcBars B{tc5::smem_addr(tail), p.error, false};
  const uint32_t tmem_slot = tc5::smem_addr(tail) + 160;
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      tc5::mbar_init(B.full(b), 1);
      tc5::mbar_init(B.empty(b), kTcEpiWarps);
    }
    for (int c = 0; c < 4; ++c) tc5::mbar_init(B.written(c), kTcEpiWarps);
    for (int r = 0; r < NR; ++r) {
      tc5::mbar_init(B.unused(r), 1);
      tc5::mbar_init(B.loaded(r), 32 * tc_load_warps(SRC));
    }
  }
  if (warp == kTcEpiWarps) tc5::tmem_alloc(tmem_slot, 512);
  tc5::fence_async_smem();
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem0 = *reinterpret_cast<volatile uint32_t*>(tail + 160);

  auto offset = [&](uint32_t e) {  // codeword offset of slot bits e
    uint32_t a = 0;
#pragma unroll
    for (int j = 0; j < kTcTileLog; ++j) a += (e >> j & 1) * p.stride[j];
    return a;
  };
  // kMidAlpha walks the columns first, so that concurrent tiles share alphas.
  auto real_tile = [&](uint32_t v) {
    if constexpr (MID == kMidAlpha)
      return (v & ((1u << p.col_log) - 1u)) * (p.n_tiles >> p.col_log) + (v >> p.col_log);
    else
      return v;
  };

  if (warp < kTcEpiWarps) {
    const uint32_t m = uint32_t(lane) | uint32_t(warp & 3) << 5, g = uint32_t(warp >> 2) << 2;
    const uint32_t ex = LX::of_m(m) | LX::of_n(g), ey = LY::of_m(m) | LY::of_n(g);
    const uint32_t tmem = tmem0 + (uint32_t(warp & 3) << 21) + 16u * g, c256 = p.c256;
    const uint32_t ring_s = tc5::smem_addr(ring);
    uint32_t u = 0;  // chunks so far
    uint32_t ring_x = 0, ring_y = uint32_t(warp & 3);  // regions of chunk 0, and of this warp's stage Y elements
    auto nothing = [] {};
    auto keep = [](int, Fr&) {};
    auto x_region = [&](int c) { const uint32_t r = ring_x + c; return ring_s + (r >= NR ? r - NR : r) * kTcRegionBytes; };
    auto x_out = [&](Fe* to, int c) { return to + offset(ex) + uint32_t(c & 1) * p.stride[LX::chunk(0)] + uint32_t(c >> 1) * p.stride[LX::chunk(1)]; };
    for (uint32_t vt = blockIdx.x; vt < p.n_tiles; vt += gridDim.x) {
      const uint32_t tile = real_tile(vt);
      const uint32_t tbase = tc_tile_base(p, tile);
      const uint32_t y_region = ring_s + ring_y * kTcRegionBytes;
      if constexpr (kTwo && HASY) {
        const uint32_t xy = LY::unit(ex);
#pragma unroll 1
        for (int c = 0; c < 4; ++c, ++u) tc_chunk<CFG, true, 2, kParts>(B, x_region(c), tmem, u, c, xy, c256, nothing, keep);
        const uint32_t yy = LY::unit(ey);
#pragma unroll 1
        for (int c = 0; c < 4; ++c, ++u) {
          if constexpr (MID == kMidAlpha) {
            const uint32_t row = tile << kTcTileLog | ey | uint32_t(c) << LY::chunk(0), rmask = (1u << p.logR) - 1u;
            uint4 al[4];
            tc_chunk<CFG, false, 2, kParts>(
                B, y_region, tmem, u, c, yy, c256,
                [&] {
#pragma unroll
                  for (int i = 0; i < 4; ++i) al[i] = __ldg(reinterpret_cast<const uint4*>(p.alpha) + ((row | LY::of_n(i)) & rmask));
                },
                [&](int i, Fr& v) { v = mul(v, unpack_fe(al[i])); });
          } else {
            Fe* mid = p.mid + tbase + offset(ey) + uint32_t(c & 1) * p.stride[LY::chunk(0)] + uint32_t(c >> 1) * p.stride[LY::chunk(1)];
            tc_chunk<CFG, false, 2, kParts>(B, y_region, tmem, u, c, yy, c256, nothing, [&](int i, Fr& v) {
              *reinterpret_cast<uint4*>(mid + offset(LY::of_n(i))) = pack_fe(v);
            });
          }
        }
      }
      if constexpr (kTwo && !HASY) {
        const uint32_t xx = LX::unit(ex);
#pragma unroll 1
        for (int c = 0; c < 4; ++c, ++u) {
          Fe* mid = x_out(p.mid + tbase, c);
          tc_chunk<CFG, true, 1, kParts>(B, x_region(c), tmem, u, c, xx, c256, nothing, [&](int i, Fr& v) {
            *reinterpret_cast<uint4*>(mid + offset(LX::of_n(i))) = pack_fe(v);
          });
        }
      }
      if constexpr (HASY) {
        const uint32_t yx = LX::unit(ey);
#pragma unroll 1
        for (int c = 0; c < 4; ++c, ++u) tc_chunk<CFG, false, 1, kParts>(B, y_region, tmem, u, c, yx, c256, nothing, keep);
      }
#pragma unroll 1
      for (int c = 0; c < 4; ++c, ++u) {
        Fe* dst = x_out(p.dst + tbase, c);
        tc_chunk<CFG, true, 0, kParts>(B, 0, tmem, u, c, 0, c256, nothing, [&](int i, Fr& v) {
          *reinterpret_cast<uint4*>(dst + offset(LX::of_n(i))) = pack_fe(v);
        });
      }
      ring_x = tc_next<NR>(ring_x);
      ring_y = tc_next<NR>(ring_y);
    }
  } else if (warp == kTcEpiWarps) {
    if (lane == 0) {
      // Every offset added stays within the descriptors' 14 address bits.
      const uint64_t desc_a = tc5::smem_desc(tc5::smem_addr(mats), 16, 1024), desc_b = tc5::smem_desc(tc5::smem_addr(ring), 4096, 1024);
      uint32_t u = 0, w = 0;  // chunks, and stages that write the tile, so far
      uint32_t r0 = 0, lap[4] = {0, 0, 0, 0};  // the tile's first region; laps of the ring at each of its four
      for (uint32_t vt = blockIdx.x; vt < p.n_tiles; vt += gridDim.x) {
        uint32_t reg[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) reg[j] = r0 + j >= NR ? r0 + j - NR : r0 + j;
#pragma unroll
        for (int s = 0; s < kStages; ++s) {
          // Stage order: X | Y X | X X | X Y Y X.
          const bool x = !HASY || (kTwo ? (s == 0 || s == 3) : s == 1);
          const bool was_x = !HASY || (kTwo && s == 1);
          const bool second = kTwo && s >= kStages / 2;
          const uint32_t a = uint32_t((x ? 0 : 1) + (second && kOther ? (HASY ? 2 : 1) : 0)) * kTcMatBytes;
          const bool last = s == kStages - 1;
#pragma unroll
          for (int c = 0; c < 4; ++c, ++u) {
            if (u >= 2) B.wait(B.empty(c & 1), (u >> 1) - 1);
            if (s > 0 && x == was_x) B.wait(B.written(c), w - 1);
            if (s == 0 && x) B.wait(B.loaded(reg[c]), lap[c]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (s > 0 && x != was_x && c == 0) B.wait(B.written(j), w - 1);
              if (s == 0 && !x && c == 0) B.wait(B.loaded(reg[j]), lap[j]);
              if (s == 0) tc5::fence_async_smem();  // the loads' writes
              tc5::fence_after_sync();
              const uint32_t b = x ? reg[c] * kTcRegionBytes + (uint32_t(j) << 13) : reg[j] * kTcRegionBytes + (uint32_t(c) << 13);
              tc5::mma_i8(tmem0 + 256u * (c & 1), desc_a + ((a + 32u * j) >> 4), desc_b + (b >> 4), tc5::idesc_i8(128, 256), j > 0);
            }
            if (last) tc5::mma_commit(B.unused(reg[c]));
            tc5::mma_commit(B.full(c & 1));
          }
          if (!last) ++w;
        }
        // Position j moves by four regions: one more lap when it wraps.
#pragma unroll
        for (int j = 0; j < 4; ++j) lap[j] += reg[j] + 4 >= NR ? 1 : 0;
        r0 = tc_next<NR>(r0);
      }
      // No MMA is in flight and no arrival on its way when the CTA ends, also
      // after a wait that gave up (the last tile's regions are four back).
      if (u > 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t r = r0 + j + NR - 4, reg = r >= NR ? r - NR : r;
          tc5::mbar_wait(B.unused(reg), (lap[j] - (reg + 4 >= NR ? 1 : 0)) & 1);
        }
        for (uint32_t i = u - 2; i < u; ++i) tc5::mbar_wait(B.full(i & 1), i >> 1 & 1);
      }
    }
    __syncwarp();
  } else {
    using LF = TcLayout<CFG, kFirstX>;
    constexpr int kLow = LX::chunk(0);  // the region's slots: kLow and the next
    const uint32_t l = warp - kTcEpiWarps - 1;
    uint32_t r = 0, lap = 0;
    auto advance = [&] {
      if (++r == NR) {
        r = 0;
        ++lap;
      }
    };
    if constexpr (SRC == kTcWeights) {
      // A region is 2048 consecutive elements: eight warp-wide loads per warp,
      // a lane two elements (slot 0), lanes slots 1..5, the load and the warp
      // slots 6..10.  A region's loads are on their way while the one before
      // is waited for and stored.
      static_assert(SRC != kTcWeights || (CFG == kTileCfg && tc_load_warps(SRC) == 4), "slots of the weight loads");
      const uint32_t e0 = uint32_t(lane) << 1 | l << 9, lu = LF::unit(e0);
      const bool aligned = (reinterpret_cast<uintptr_t>(p.src) + p.src_base * sizeof(Wt)) % 16 == 0;
      uint4 raw[8];
      auto fetch = [&](uint32_t tile, uint32_t c) {
        const uint64_t first = (uint64_t(tile) << kTcTileLog) + (c << kLow);
        const bool wide = aligned && p.src_base + uint64_t(kC) * (first + 2048) <= p.active;
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) raw[i] = tc_weights(p, first + (e0 | i << 6), wide);
      };
      if (blockIdx.x < p.n_tiles) fetch(blockIdx.x, 0);
      for (uint32_t vt = blockIdx.x; vt < p.n_tiles; vt += gridDim.x) {
#pragma unroll 1
        for (uint32_t c = 0; c < 4; ++c, advance()) {
          if (lap > 0) B.wait(B.unused(r), lap - 1);
          const uint32_t to = tc5::smem_addr(ring) + r * kTcRegionBytes;
#pragma unroll
          for (uint32_t i = 0; i < 8; ++i) {
            tc5::store_shared(to + ((lu ^ LF::unit(i << 6)) << 4), pack_weights(make_uint2(raw[i].x, raw[i].y)));
            tc5::store_shared(to + ((lu ^ LF::unit(i << 6 | 1)) << 4), pack_weights(make_uint2(raw[i].z, raw[i].w)));
          }
          tc5::mbar_arrive(B.loaded(r));
          if (c < 3) fetch(vt, c + 1);
          else if (vt + gridDim.x < p.n_tiles) fetch(vt + gridDim.x, 0);
        }
      }
    } else {
      // A region: 32 warp-wide copies per warp; lanes are slots 0..4, the warp
      // and the copy the other slots without the region's.
      auto slots = [](uint32_t i) { return (i & ((1u << (kLow - 5)) - 1u)) << 5 | i >> (kLow - 5) << (kLow + 2); };
      const uint32_t e0 = uint32_t(lane) | slots(l << 5);
      const uint32_t lu = LF::unit(e0), lo = SRC == kTcElements ? offset(e0) : e0;
      for (uint32_t vt = blockIdx.x; vt < p.n_tiles; vt += gridDim.x) {
        const uint32_t tile = real_tile(vt);
#pragma unroll 1
        for (uint32_t c = 0; c < 4; ++c, advance()) {
          if (lap > 0) B.wait(B.unused(r), lap - 1);
          uint4* to = reinterpret_cast<uint4*>(ring + r * kTcRegionBytes);
          const Fe* src = static_cast<const Fe*>(p.src) +
                          (SRC == kTcLinear ? (tile << kTcTileLog) + (lo | c << kLow)
                                            : tc_tile_base(p, tile) + lo + (c & 1) * p.stride[kLow] + (c >> 1) * p.stride[kLow + 1]);
#pragma unroll
          for (int i = 0; i < 32; ++i) cp_async16(to + (lu ^ LF::unit(slots(i))), src + (SRC == kTcLinear ? slots(i) : offset(slots(i))));
          tc5::mbar_arrive_copies(B.loaded(r));
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == kTcEpiWarps) tc5::tmem_free(tmem0, 512);
}

}  // namespace QFD_NS
