// Device arithmetic for F_65521 and F_65521[X]/(X^8 - 17).
//
// Storage: 8 canonical u16 coefficients = 16 bytes, moved as one uint4
// (one 128-bit load/store per element).  Arithmetic unpacks to 32-bit
// registers.  Reductions use 2^16 = 15 (mod p) twice, the same
// pseudo-Mersenne identity as Prime65521::reduce_u32 (qafold_short.rs:336-346);
// results are canonical, so they match the host field bit for bit.
#pragma once
#include <cstdint>

// Host-callable too, so the arithmetic can be checked against the host field on a CPU.
#define QFD_HD __host__ __device__ __forceinline__

namespace qfd {

constexpr uint32_t P = 65521u;
constexpr int kC = 8;   // coefficients per element
using Wt = int8_t;      // one BVA entry

struct __align__(16) Fe {
  uint16_t c[8];
};

// Register form: eight canonical coefficients in 32-bit lanes.
struct Fr {
  uint32_t c[8];
};

QFD_HD uint32_t red32(uint32_t v) {
  uint32_t f = (v & 0xffffu) + 15u * (v >> 16);
  f = (f & 0xffffu) + 15u * (f >> 16);
  return f >= P ? f - P : f;
}
QFD_HD uint32_t red64(uint64_t v) {  // v < 2^48
  uint64_t f = (v & 0xffffu) + 15ull * (v >> 16);
  uint32_t g = uint32_t((f & 0xffffu) + 15ull * (f >> 16));
  return red32(g);
}
QFD_HD uint32_t umin32(uint32_t a, uint32_t b) { return a < b ? a : b; }
QFD_HD uint32_t addp(uint32_t a, uint32_t b) { uint32_t s = a + b; return s >= P ? s - P : s; }
QFD_HD uint32_t subp(uint32_t a, uint32_t b) { return a >= b ? a - b : a + P - b; }
// Four unsigned byte products added to c, and a byte permute (host forms for
// the CPU check of this header).
QFD_HD uint32_t dp4u(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 610
  return __dp4a(a, b, c);
#else
  for (int i = 0; i < 32; i += 8) c += ((a >> i) & 0xffu) * ((b >> i) & 0xffu);
  return c;
#endif
}
QFD_HD uint32_t bytes(uint32_t a, uint32_t b, uint32_t sel) {
#if defined(__CUDA_ARCH__)
  return __byte_perm(a, b, sel);
#else
  const uint64_t v = uint64_t(b) << 32 | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; ++i) r |= uint32_t(v >> (8 * (sel >> (4 * i) & 7)) & 0xffu) << (8 * i);
  return r;
#endif
}

QFD_HD Fr load(const Fe* p) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  Fr r;
  r.c[0] = u.x & 0xffffu; r.c[1] = u.x >> 16;
  r.c[2] = u.y & 0xffffu; r.c[3] = u.y >> 16;
  r.c[4] = u.z & 0xffffu; r.c[5] = u.z >> 16;
  r.c[6] = u.w & 0xffffu; r.c[7] = u.w >> 16;
  return r;
}
QFD_HD void store(Fe* p, const Fr& r) {
  uint4 u;
  u.x = r.c[0] | (r.c[1] << 16);
  u.y = r.c[2] | (r.c[3] << 16);
  u.z = r.c[4] | (r.c[5] << 16);
  u.w = r.c[6] | (r.c[7] << 16);
  *reinterpret_cast<uint4*>(p) = u;
}
QFD_HD Fr zero() { Fr r; for (int i = 0; i < 8; ++i) r.c[i] = 0; return r; }
QFD_HD Fr add(const Fr& a, const Fr& b) { Fr r; for (int i = 0; i < 8; ++i) r.c[i] = addp(a.c[i], b.c[i]); return r; }
QFD_HD Fr sub(const Fr& a, const Fr& b) { Fr r; for (int i = 0; i < 8; ++i) r.c[i] = subp(a.c[i], b.c[i]); return r; }
// v < 2^40 to canonical: two 2^16 = 15 folds (< 2^28 + 2^16, then < 2p) and
// one conditional subtraction.
QFD_HD uint32_t red40(uint64_t v) {
  uint32_t f = uint32_t(v & 0xffffu) + 15u * uint32_t(v >> 16);
  f = (f & 0xffffu) + 15u * (f >> 16);
  return f >= P ? f - P : f;
}
// A signed v with |v| < 2^62: adding kBias (the multiple of p just above
// 2^62) gives an unsigned value below 2^64 with the same residue; two folds
// of 2^16 = 15 bring it below 2^40 for red40.
constexpr uint64_t kBias = ((uint64_t(1) << 62) / P + 1) * P;
QFD_HD uint32_t red_signed(int64_t v) {
  uint64_t u = uint64_t(v) + kBias;
  u = (u & 0xffffu) + 15u * (u >> 16);
  u = (u & 0xffffu) + 15u * (u >> 16);
  return red40(u);
}
// The product's output coefficients, raw: coefficient k is the sum over i of
// a_i w_(k - i), w_j = b_j and, for the wrap-around X^8 = 17, w_(j - 8) = 17 b_j
// mod p.  All operands are 16 bits, so their byte planes multiply by dp4a,
// four products each: with s0, s1, s2 the sums of the low-low, mixed and
// high-high byte products, the coefficient is s0 + 2^8 s1 + 2^16 s2, and 2^16
// = 15 keeps it in 32 bits (below 2^28.1).  64 dp4a take 1.40 clocks per
// product and SM with the reductions (measured on B200, operands in
// registers); 64 widening multiply-adds, which issue at half that rate each,
// took 2.04.
struct Raw {
  uint32_t c[8];
};
QFD_HD Raw mul_raw(const Fr& a, const Fr& b) {
  // Bytes a_0..a_3 and a_4..a_7, low and high.
  uint32_t al[2], ah[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t x = bytes(a.c[4 * i], a.c[4 * i + 1], 0x5410), y = bytes(a.c[4 * i + 2], a.c[4 * i + 3], 0x5410);
    al[i] = bytes(x, y, 0x6420);
    ah[i] = bytes(x, y, 0x7531);
  }
  // w_7, w_6, .., w_0, w_-1, .., w_-8 as bytes.  A loop's fixed factor goes
  // second, so that these are formed once.
  uint32_t wl[4], wh[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = b.c[7 - ((4 * i + j) & 7)];
      if (i >= 2) {
        v[j] *= 17u;
        v[j] -= (v[j] >> 16) * P;
        v[j] = umin32(v[j], v[j] - P);
      }
    }
    const uint32_t x = bytes(v[0], v[1], 0x5410), y = bytes(v[2], v[3], 0x5410);
    wl[i] = bytes(x, y, 0x6420);
    wh[i] = bytes(x, y, 0x7531);
  }
  Raw r;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    // The window w_k, w_(k - 1), .., w_(k - 7).
    const int q = (7 - k) >> 2, sh = (7 - k) & 3;
    const uint32_t sel = sh == 1 ? 0x4321u : (sh == 2 ? 0x5432u : 0x6543u);
    const uint32_t l0 = sh ? bytes(wl[q], wl[q + 1], sel) : wl[q], l1 = sh ? bytes(wl[q + 1], wl[q + 2], sel) : wl[q + 1];
    const uint32_t h0 = sh ? bytes(wh[q], wh[q + 1], sel) : wh[q], h1 = sh ? bytes(wh[q + 1], wh[q + 2], sel) : wh[q + 1];
    const uint32_t s0 = dp4u(al[1], l1, dp4u(al[0], l0, 0u)), s2 = dp4u(ah[1], h1, dp4u(ah[0], h0, 0u));
    const uint32_t s1 = dp4u(al[1], h1, dp4u(al[0], h0, dp4u(ah[1], l1, dp4u(ah[0], l0, 0u))));
    r.c[k] = s2 * 15u + s0 + s1 * 256u;
  }
  return r;
}
QFD_HD Fr mul(const Fr& a, const Fr& b) {
  const Raw r = mul_raw(a, b);
  Fr out;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t f = r.c[k] - (r.c[k] >> 16) * P;  // below 2^16 + 15 * 2^12.1 < 2p
    out.c[k] = umin32(f, f - P);
  }
  return out;
}
// Lazy sums of products: a raw product is below 2^28.1 per coefficient, so a
// 64-bit accumulator takes 2^24 products with room to spare; it is reduced
// once at the end (two folds of 2^16 = 15 bring any u64 below 2^40, then
// red40).
struct Acc {
  uint64_t c[8];
};
QFD_HD Acc acc_zero() { Acc r; for (int k = 0; k < 8; ++k) r.c[k] = 0; return r; }
QFD_HD void mul_acc(Acc& r, const Fr& a, const Fr& b) {
  const Raw t = mul_raw(a, b);
#pragma unroll
  for (int k = 0; k < 8; ++k) r.c[k] += t.c[k];
}
QFD_HD Fr acc_reduce(const Acc& r) {
  Fr out;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    uint64_t v = (r.c[k] & 0xffffu) + 15u * (r.c[k] >> 16);
    v = (v & 0xffffu) + 15u * (v >> 16);
    out.c[k] = red40(v);
  }
  return out;
}
QFD_HD Fr mul_base(const Fr& a, uint32_t s) {
  Fr r;
  for (int i = 0; i < 8; ++i) r.c[i] = red32(a.c[i] * s);
  return r;
}
// Σ of kC products of canonical values (< 2^35) to canonical.
QFD_HD uint32_t red_sum(uint64_t v) { return red64(v); }
QFD_HD Fr unpack_fe(uint4 u) {
  Fr v;
  v.c[0] = u.x & 0xffffu; v.c[1] = u.x >> 16; v.c[2] = u.y & 0xffffu; v.c[3] = u.y >> 16;
  v.c[4] = u.z & 0xffffu; v.c[5] = u.z >> 16; v.c[6] = u.w & 0xffffu; v.c[7] = u.w >> 16;
  return v;
}
QFD_HD uint32_t pack16(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __byte_perm(a, b, 0x5410);
#else
  return a | (b << 16);
#endif
}
QFD_HD uint4 pack_fe(const Fr& r) {
  return make_uint4(pack16(r.c[0], r.c[1]), pack16(r.c[2], r.c[3]), pack16(r.c[4], r.c[5]), pack16(r.c[6], r.c[7]));
}

// Planar transform tiles use lazy reduction: a value entering level l of a
// pass is below tile_bound(l) = 2^l p, a difference is formed as a + 2^l p - b,
// so twelve levels stay below 2^28 and tile_final reduces once per pass.
QFD_HD uint32_t tile_bound(int lvl) { return P << lvl; }
QFD_HD void bfly_wht(uint32_t& lo, uint32_t& hi, uint32_t B) {
  const uint32_t a = lo, b = hi;
  lo = a + b;
  hi = a + B - b;
}
QFD_HD void bfly_mobius(uint32_t lo, uint32_t& hi, uint32_t B) { hi = hi + B - lo; }
// Values below 2^28 (at most twelve lazy levels) to canonical form.
QFD_HD uint32_t tile_final(uint32_t v) {
  const uint32_t f = (v & 0xffffu) + 15u * (v >> 16);  // < 2^16 + 15 * 2^12 < 2p
  return f >= P ? f - P : f;
}

// Limb sums of the tensor-core transforms: s[2i] and s[2i + 1] hold (as s32)
// sums of at most 128 signed terms of coefficient i's low and high byte.  The
// coefficient t = s[2i] + 256 s[2i + 1] is within 128 (p - 1) of zero; adding
// 128 p makes it an unsigned value below 2^24, one fold of 2^16 = 15 (as a
// multiply-add, t - 65521 (t >> 16)) brings it below 2 p.
#if defined(__CUDACC__)
__device__ __forceinline__ Fr limb_sums(const uint32_t (&s)[16], uint32_t c256) {
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t t = s[2 * i + 1] * c256 + (s[2 * i] + 128u * P);
    const uint32_t f = t - (t >> 16) * P;
    r.c[i] = __viaddmin_u32(f, 0u - P, f);
  }
  return r;
}
#endif

// small signed integer -> canonical F_65521 (field.rs:24-26)
QFD_HD uint32_t small(int v) { return v < 0 ? uint32_t(v + int(P)) : uint32_t(v); }
// Eight signed 8-bit weights (8 bytes) to the packed element.
QFD_HD Fr weights_to_fr(uint2 raw) {
  Fr r;
#pragma unroll
  for (int k = 0; k < 8; ++k) r.c[k] = small(int(int8_t(((k < 4 ? raw.x : raw.y) >> (8 * (k & 3))) & 0xffu)));
  return r;
}

// The same packed: bytes sign-extended in 16-bit pairs, less 15 where negative
// (v + p = v - 15 mod 2^16, and no borrow leaves the half).
#if defined(__CUDACC__)
__device__ __forceinline__ uint4 pack_weights(uint2 raw) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t b = i < 2 ? raw.x : raw.y;
    uint32_t v, sign;  // a selector nibble of 8 + j replicates byte j's sign
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(v) : "r"(b), "r"(i & 1 ? 0xb3a2u : 0x9180u));
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(sign) : "r"(b), "r"(i & 1 ? 0xbbaau : 0x9988u));
    w[i] = v - (sign & 0x000f000fu);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
#endif

}  // namespace qfd
