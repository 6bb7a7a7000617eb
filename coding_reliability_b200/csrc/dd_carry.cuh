// dd_carry.cuh — packed distance histograms in registers and the tables they are
// added to, shared by the residue-pair kernels (dd_carry.cu, dd_carry_rows.cu).
#pragma once
#include "dd_carry.h"

namespace dd {
namespace {

// Distances a table holds: up to 24 from the enumerated bits, up to 28 (bins that a
// packed word can name) from the window and the high words.
constexpr int kTabRows = 56;
constexpr int kTabBytes = kTabRows * 128;  // one column per lane

// Counts of bins 8j + 2i (e[j], byte i) and 8j + 2i + 1 (o[j], byte i).
struct H8 {
  uint32_t e[3], o[3];
};
// Counts of bins 8j + m (low half of pm[j]) and 8j + 4 + m (high half).
struct H16 {
  uint32_t p0[4], p1[3], p2[3], p3[3];
};

__device__ __forceinline__ void zero(H16& h) {
#pragma unroll
  for (int j = 0; j < 3; ++j) h.p0[j] = h.p1[j] = h.p2[j] = h.p3[j] = 0;
  h.p0[3] = 0;
}

// x + z y
__device__ __forceinline__ H8 add_z(const H8& x, const H8& y) {
  H8 r;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.e[j] = x.e[j] + (j ? __funnelshift_l(y.o[j - 1], y.o[j], 8) : y.o[0] << 8);
    r.o[j] = x.o[j] + y.e[j];
  }
  return r;
}
__device__ __forceinline__ H16 add_z(const H16& x, const H16& y) {
  H16 r;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.p0[j] = x.p0[j] + (j ? __funnelshift_l(y.p3[j - 1], y.p3[j], 16) : y.p3[0] << 16);
    r.p1[j] = x.p1[j] + y.p0[j];
    r.p2[j] = x.p2[j] + y.p1[j];
    r.p3[j] = x.p3[j] + y.p2[j];
  }
  r.p0[3] = x.p0[3] + (y.p3[2] >> 16);
  return r;
}
__device__ __forceinline__ H8 add(const H8& x, const H8& y) {
  H8 r;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.e[j] = x.e[j] + y.e[j];
    r.o[j] = x.o[j] + y.o[j];
  }
  return r;
}
__device__ __forceinline__ H16 add(const H16& x, const H16& y) {
  H16 r;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.p0[j] = x.p0[j] + y.p0[j];
    r.p1[j] = x.p1[j] + y.p1[j];
    r.p2[j] = x.p2[j] + y.p2[j];
    r.p3[j] = x.p3[j] + y.p3[j];
  }
  r.p0[3] = x.p0[3] + y.p0[3];
  return r;
}
__device__ __forceinline__ H16 widen(const H8& h) {
  H16 r;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.p0[j] = h.e[j] & 0x00FF00FFu;
    r.p1[j] = h.o[j] & 0x00FF00FFu;
    r.p2[j] = (h.e[j] >> 8) & 0x00FF00FFu;
    r.p3[j] = (h.o[j] >> 8) & 0x00FF00FFu;
  }
  r.p0[3] = 0;
  return r;
}
// One column's histogram in a shared exchange row: 24 bytes (8-bit counts) or 48
// (16-bit counts below the last level, whose bins stop at 23), at strides that
// make the vector accesses conflict-free.
__device__ __forceinline__ void put(uint8_t* row, int c, const H8& h) {
  uint2* p = reinterpret_cast<uint2*>(row + c * 24);
  p[0] = make_uint2(h.e[0], h.e[1]);
  p[1] = make_uint2(h.e[2], h.o[0]);
  p[2] = make_uint2(h.o[1], h.o[2]);
}
__device__ __forceinline__ void get(const uint8_t* row, int c, H8& h) {
  const uint2* p = reinterpret_cast<const uint2*>(row + c * 24);
  const uint2 x = p[0], y = p[1], w = p[2];
  h.e[0] = x.x; h.e[1] = x.y; h.e[2] = y.x; h.o[0] = y.y; h.o[1] = w.x; h.o[2] = w.y;
}
__device__ __forceinline__ void put(uint8_t* row, int c, const H16& h) {
  uint4* p = reinterpret_cast<uint4*>(row + c * 48);
  p[0] = make_uint4(h.p0[0], h.p0[1], h.p0[2], h.p1[0]);
  p[1] = make_uint4(h.p1[1], h.p1[2], h.p2[0], h.p2[1]);
  p[2] = make_uint4(h.p2[2], h.p3[0], h.p3[1], h.p3[2]);
}
__device__ __forceinline__ void get(const uint8_t* row, int c, H16& h) {
  const uint4* p = reinterpret_cast<const uint4*>(row + c * 48);
  const uint4 x = p[0], y = p[1], w = p[2];
  h.p0[0] = x.x; h.p0[1] = x.y; h.p0[2] = x.z; h.p1[0] = x.w;
  h.p1[1] = y.x; h.p1[2] = y.y; h.p2[0] = y.z; h.p2[1] = y.w;
  h.p2[2] = w.x; h.p3[0] = w.y; h.p3[1] = w.z; h.p3[2] = w.w;
  h.p0[3] = 0;
}

// The first level from the four high-word distances: z^ha + z^hd + z (z^hb + z^hc).
// Each distance adds 1 to a nibble (two nibbles per byte: bins 8 apart), a
// distance of 16 to the count x.
struct Nibbles {
  uint32_t e = 0, o = 0, x = 0;
  __device__ __forceinline__ void count(uint32_t h) {
    const uint32_t one = 1u << (((h << 2) & 24u) | ((h >> 1) & 4u));
    if (h & 1u) o += one;
    else e += one;
    x += h >> 4;
  }
  __device__ __forceinline__ H8 bytes() const {
    const uint32_t ev = e - x;  // a distance of 16 was counted in bin 0, too
    return H8{{ev & 0x0F0F0F0Fu, (ev >> 4) & 0x0F0F0F0Fu, x}, {o & 0x0F0F0F0Fu, (o >> 4) & 0x0F0F0F0Fu, 0u}};
  }
};
__device__ __forceinline__ H8 first_level(uint32_t ra, uint32_t rb, uint32_t ca, uint32_t cb) {
  Nibbles same, cross;
  same.count(__popc(ra ^ ca));
  same.count(__popc(rb ^ cb));
  cross.count(__popc(ra ^ cb));
  cross.count(__popc(rb ^ ca));
  return add_z(same.bytes(), cross.bytes());
}

// a v mod A for a < A < 2^16 (32-bit divisions only)
__device__ __forceinline__ uint32_t mul_mod(uint32_t a, uint32_t v, uint32_t A) { return a * (v % A) % A; }
__device__ __forceinline__ uint32_t sub_mod(uint32_t x, uint32_t d, uint32_t A) { return x >= d ? x - d : x + A - d; }

template <int kOffset>
__device__ __forceinline__ void red_add(uint32_t addr, uint32_t x) {
  asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(addr), "n"(kOffset), "r"(x) : "memory");
}

// Adds f x (the counts of h) to a lane's table column, bin d at at + 128 d.
// kProduct: f is 1; 32-bit products; products of up to 48 bits, whose low 16 bits go
// to the first table and the rest to the one two tables on.
enum Product { kOne, kNarrow, kWideProduct };
template <int kProduct, int kBin>
__device__ __forceinline__ void add_bin(uint32_t at, uint32_t f, uint32_t x) {
  if constexpr (kProduct == kWideProduct) {
    const unsigned long long p = (unsigned long long)f * x;
    red_add<kBin * 128>(at, (uint32_t)p & 0xFFFFu);
    red_add<kBin * 128 + 2 * kTabBytes>(at, (uint32_t)(p >> 16));
  } else {
    red_add<kBin * 128>(at, kProduct == kNarrow ? f * x : x);
  }
}
template <int kProduct, int kBin>
__device__ __forceinline__ void add_halves(uint32_t at, uint32_t f, uint32_t w) {
  if (w) {
    add_bin<kProduct, kBin>(at, f, w & 0xFFFFu);
    add_bin<kProduct, kBin + 4>(at, f, w >> 16);
  }
}
template <int kProduct>
__device__ __forceinline__ void add_hist(uint32_t at, uint32_t f, const H16& h) {
  add_halves<kProduct, 0>(at, f, h.p0[0]); add_halves<kProduct, 1>(at, f, h.p1[0]);
  add_halves<kProduct, 2>(at, f, h.p2[0]); add_halves<kProduct, 3>(at, f, h.p3[0]);
  add_halves<kProduct, 8>(at, f, h.p0[1]); add_halves<kProduct, 9>(at, f, h.p1[1]);
  add_halves<kProduct, 10>(at, f, h.p2[1]); add_halves<kProduct, 11>(at, f, h.p3[1]);
  add_halves<kProduct, 16>(at, f, h.p0[2]); add_halves<kProduct, 17>(at, f, h.p1[2]);
  add_halves<kProduct, 18>(at, f, h.p2[2]); add_halves<kProduct, 19>(at, f, h.p3[2]);
  add_halves<kProduct, 24>(at, f, h.p0[3]);
}

// ---------------------------------------------------------------- host side
inline uint32_t inverse_pow2(uint32_t e, uint32_t A) {  // 2^-e mod A, A odd
  uint64_t x = 1 % A;
  const uint64_t half = (A + 1) / 2 % A;
  for (uint32_t i = 0; i < e; ++i) x = x * half % A;
  return (uint32_t)x;
}

inline uint32_t odd_part(uint64_t A) {
  while (A && !(A & 1)) A >>= 1;
  return (uint32_t)A;
}
inline uint32_t bits_of(uint32_t x) {
  uint32_t n = 0;
  for (; x; x >>= 1) ++n;
  return n;
}

}  // namespace
}  // namespace dd
