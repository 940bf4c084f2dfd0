// One 32-element block per thread, in registers: the arithmetic that every codec kernel shares.
//
// Integers as subnormal floats.  A whole number k with |k| < 2^24 is held as the float k * 2^-149, whose bits
// ARE sign and magnitude of k (for exponents 0 and 1 the significand field counts in steps of 2^-149).
// Additions and subtractions of such numbers are exact on the fp32 pipe, take no conversion, and leave the
// sign-magnitude form that the stream stores.  On sm_100 integer add, logic, shift and byte-permute issue at
// half rate on one pipe and a float -> int conversion at an eighth; fp32 add, multiply and fma do not touch
// that pipe.  Quantise + Lorenzo of a block: 278 cycles a warp and scheduler in this form against 422 with
// __float2int_rz and int32 differences (B200, isolated loop).  Blocks outside the range take the int32 path.
#pragma once
#include "hc_bitplane.h"
#include "hc_device.cuh"

namespace hc {
namespace dev {

__device__ __forceinline__ float as_f(uint32_t u) { return __uint_as_float(u); }
__device__ __forceinline__ uint32_t as_u(float f) { return __float_as_uint(f); }
constexpr uint32_t kMsb = 0x80000000u;

// 32-bit shared-memory load by shared-window address (a generic pointer would turn it into a generic load)
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
// (a & b) | c in one operation, with b and c kept from being split into two immediates
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// ---- quantiser ----------------------------------------------------------------------------------
__device__ __forceinline__ int32_t quantise(float x, float recip) {
  float t = __fmul_rn(x, recip);  // two roundings: the stream is defined without FMA contraction
  float u = __fadd_rn(t, 0.5f);
  return __float2int_rz(u) - ((t >= -0.5f) ? 0 : 1);
}
// The same value as a subnormal.  u = t + 0.5 is exact for t < -0.5, so "t < -0.5" is the sign of u; the
// multiplication by 2^-149 truncates towards zero and keeps the sign, whose bit then is the "minus one"
// (one more in magnitude).  Equal to quantise() for every float with |x * recip| < 2^24 (checked over all of
// them); beyond that the result is only good for being recognised as out of range.
__device__ __forceinline__ float quantise_sub(float x, float recip) {
  const float u = __fadd_rn(__fmul_rn(x, recip), 0.5f);
  const uint32_t z = as_u(__fmul_rz(u, as_f(1u)));
  return as_f(z + (z >> 31));
}

// ---- tile rows in shared memory, 128-byte TMA swizzle ----------------------------------------------
// 16-byte unit c of row `row` sits at unit c ^ (row & 7); `rows` must be 1024-byte aligned, so that the address
// of a unit is one xor away from the row's
__device__ __forceinline__ uint32_t swizzled_row(const uint8_t* rows, int row) {
  return (smem_u32(rows) + (uint32_t)row * 128u) | (((uint32_t)row & 7u) << 4);
}
__device__ __forceinline__ void load_row_swizzled(const uint8_t* rows, int row, uint32_t (&w)[32]) {
  const uint32_t r = swizzled_row(rows, row);
#pragma unroll
  for (int c = 0; c < 8; ++c)
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[4 * c]), "=r"(w[4 * c + 1]), "=r"(w[4 * c + 2]), "=r"(w[4 * c + 3])
                 : "r"(r ^ (c << 4))
                 : "memory");
}
__device__ __forceinline__ void store_row_swizzled(uint8_t* rows, int row, const uint32_t (&w)[32]) {
  const uint32_t r = swizzled_row(rows, row);
#pragma unroll
  for (int c = 0; c < 8; ++c)
    asm volatile("st.shared.v4.u32 [%4], {%0, %1, %2, %3};" ::"r"(w[4 * c]), "r"(w[4 * c + 1]), "r"(w[4 * c + 2]),
                 "r"(w[4 * c + 3]), "r"(r ^ (c << 4))
                 : "memory");
}
// plain-load path (unaligned base, tiny inputs) and the ragged last row
__device__ __forceinline__ void load_row_global(const uint32_t* base, uint64_t n, uint64_t row, uint32_t (&w)[32]) {
  uint64_t o = row * kBlock;
#pragma unroll
  for (int i = 0; i < 32; ++i) w[i] = (o + i < n) ? __ldg(base + o + i) : 0u;
}

// ---- payload lengths ----------------------------------------------------------------------------------
// sum of payload_len over the four rate bytes of a word
__device__ __forceinline__ uint32_t payload_len4(uint32_t r4) {
  const uint32_t F = r4 & 0x1f1f1f1fu, outl = r4 & 0x80808080u;
  const uint32_t live = ((F + 0x7f7f7f7fu) | r4) & 0x80808080u;          // F > 0 or outlier layout
  const uint32_t extra = (r4 >> 5) & ((outl >> 7) * 3u);                  // outlier bytes - 1, per byte
  return 4u * __dp4a(F, 0x01010101u, 0u) + 4u * __popc(live) + __popc(outl) + __dp4a(extra, 0x01010101u, 0u);
}

// ---- stream -> block --------------------------------------------------------------------------------
// Reads the payload of the block with rate byte `rate` at byte `pos` of a staged stream: planes into T[0..W-1]
// (zero at and above F), the sign map with element i at bit 31 - i, |d0| of an outlier block (else 0).  Every
// word is rebuilt from two neighbours by a funnel shift, whatever the block's alignment: with outlier blocks
// about, the lanes of a warp have all four alignments, and a second path for aligned blocks ran on top.
// Blocks without payload give zeros; up to 4 W + 8 bytes behind the payload are read (and ignored).
template <int W>
__device__ __forceinline__ void read_planes(const uint8_t* buf, uint32_t pos, uint32_t rate, bool any_outlier,
                                            uint32_t& sign, uint32_t& a0, uint32_t (&T)[32]) {
  const uint32_t F = rate & 31u;
  uint32_t p2 = pos;
  a0 = 0;
  if (any_outlier && (rate & 0x80u)) {
    const uint32_t nout = ((rate >> 5) & 3u) + 1u;
    const uint32_t wa = smem_u32(buf) + (pos & ~3u);
    a0 = __funnelshift_r(lds32(wa), lds32(wa + 4u), 8u * (pos & 3u)) & (0xffffffffu >> (32u - 8u * nout));
    p2 += nout;
  }
  const uint32_t sh = 8u * (p2 & 3u);
  const uint32_t wp = smem_u32(buf) + (p2 & ~3u);
  // every lane loads as many words as the widest block of the warp has (no branches; words behind the block's
  // own payload are dropped)
  uint32_t word[W + 2];
#pragma unroll
  for (int j = 0; j < W + 2; ++j) word[j] = lds32(wp + 4 * j);
  sign = __byte_perm(__funnelshift_r(word[0], word[1], sh), 0, 0x0123);
#pragma unroll
  for (int j = 1; j <= W; ++j) {
    const uint32_t x = __funnelshift_r(word[j], word[j + 1], sh);
    T[j - 1] = (uint32_t)j <= F ? x : 0u;
  }
}

// planes -> rows: on return T[i ^ 7] = |d_i|
template <int W>
__device__ __forceinline__ void rows_of_block(uint32_t (&T)[32], uint32_t rate, uint32_t a0) {
  if (W == 0) {
#pragma unroll
    for (int i = 0; i < 32; ++i) T[i] = 0;
  } else {
    rows_from_planes<W == 0 ? 4 : W>(T);
  }
  if (rate & 0x80u) T[7] = a0 & 0x7fffffffu;
}

// staged payload -> rows; W (plane_width of the largest F of the warp) is warp-uniform
__device__ __forceinline__ void decode_rows(const uint8_t* buf, uint32_t pos, uint32_t rate, int W, uint32_t& sign,
                                            uint32_t& a0, uint32_t (&T)[32]) {
  const bool outl = __any_sync(0xffffffffu, rate & 0x80u);
  switch (W) {
    case 0: read_planes<0>(buf, pos, rate, outl, sign, a0, T); rows_of_block<0>(T, rate, a0); break;
    case 4: read_planes<4>(buf, pos, rate, outl, sign, a0, T); rows_of_block<4>(T, rate, a0); break;
    case 8: read_planes<8>(buf, pos, rate, outl, sign, a0, T); rows_of_block<8>(T, rate, a0); break;
    case 12: read_planes<12>(buf, pos, rate, outl, sign, a0, T); rows_of_block<12>(T, rate, a0); break;
    case 16: read_planes<16>(buf, pos, rate, outl, sign, a0, T); rows_of_block<16>(T, rate, a0); break;
    default: read_planes<32>(buf, pos, rate, outl, sign, a0, T); rows_of_block<32>(T, rate, a0); break;
  }
}

// 2^126 with the sign of element i: |d_i| * 2^-149 (the row as it stands, read as a float) times this is
// d_i * 2^-23, which fma accumulates exactly while the sum stays below 2^24 steps
__device__ __forceinline__ float sign_scale(uint32_t sign, int i) { return as_f(and_or(sign << i, kMsb, 0x7e800000u)); }
// |d_i| and sign -> d_i as a subnormal
__device__ __forceinline__ float signed_sub(uint32_t mag, uint32_t sign, int i) { return as_f(mag ^ ((sign << i) & kMsb)); }

}  // namespace dev
}  // namespace hc
