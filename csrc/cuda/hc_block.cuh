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
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
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
// The same as subnormals, two values at a time: the packed fp32 operations of sm_100 do the work of two in one issue slot
// (64 instructions less a block than with single ones).  With u = t + 0.5, exact for t < -0.5, "t < -0.5" is the sign of u and
// the quantised value is u rounded down, one less still where u is a negative whole number.  u + u * 2^-24 rounded down is u
// itself where u >= 0 and the next float below where u < 0, and that times 2^-149 rounded down is the value.  Equal to quantise()
// for every float with |x * recip| < 2^24 (checked over all of them at six scales); beyond that the result is only good
// for being recognised as out of range.
// `one`: 1.0f that the compiler does not know to be one.  The assembler contracts a packed multiplication and a packed addition
// that follows it into one operation with one rounding, whatever the rounding modifiers say; a multiplication by an unknown
// value keeps the two apart.
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b));
  return v;
}
__device__ __forceinline__ void unpack2(uint64_t v, uint32_t& a, uint32_t& b) { asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t twice(float f) { return pack2(as_u(f), as_u(f)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
__device__ __forceinline__ void quantise_sub2(uint32_t& a, uint32_t& b, uint64_t recip, uint64_t one) {
  const uint64_t u = fma2(mul2(pack2(a, b), recip), one, twice(0.5f));
  uint64_t v, z;
  asm("fma.rm.f32x2 %0, %1, %2, %1;" : "=l"(v) : "l"(u), "l"(twice(0x1p-24f)));
  asm("mul.rm.f32x2 %0, %1, %2;" : "=l"(z) : "l"(v), "l"(pack2(1u, 1u)));
  unpack2(z, a, b);
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
// plain-load path (unaligned base, tiny inputs) and the ragged last row.  Coherent loads, not __ldg: in an allreduce in
// place a step that is already running writes to the array that this one reads.
__device__ __forceinline__ void load_row_global(const uint32_t* base, uint64_t n, uint64_t row, uint32_t (&w)[32]) {
  uint64_t o = row * kBlock;
#pragma unroll
  for (int i = 0; i < 32; ++i) w[i] = (o + i < n) ? base[o + i] : 0u;
}

// ---- payload lengths ----------------------------------------------------------------------------------
// sum of payload_len over the four rate bytes of a word
__device__ __forceinline__ uint32_t payload_len4(uint32_t r4) {
  const uint32_t F = r4 & 0x1f1f1f1fu, outl = r4 & 0x80808080u;
  const uint32_t live = ((F + 0x7f7f7f7fu) | r4) & 0x80808080u;          // F > 0 or outlier layout
  const uint32_t extra = (r4 >> 5) & ((outl >> 7) * 3u);                  // outlier bytes - 1, per byte
  return 4u * __dp4a(F, 0x01010101u, 0u) + 4u * __popc(live) + __popc(outl) + __dp4a(extra, 0x01010101u, 0u);
}

// element 0 of a block in the order of the stream's words
constexpr uint32_t kFirst = 0x80u;

// Which of the first 16 planes a block of F planes has: all ones or zero for each, a row of 16 words for every F.  Comparing and
// selecting takes two operations a plane of the half-rate pipe; with a mask from shared memory it is one, in sums together with the
// exclusive or with the sign (decode of 64 MB 22.5 us, 21.2 this way, of 256 MB 61.8 and 60.9; four streams of 256 MB added 143.5 and
// 138.8; the decode of an allreduce step of 64 MB at 8 ranks 33.1 and 32.0).  Not in the add of one stream and fp32: of 64 MB 38.6 us,
// 38.4 with masks, but of 4 MB 7.7 and 7.8, for the time that the rows take at the start.  Nor for blocks of 13 to 16 planes in the decode
// of one stand-alone stream (a random walk of 256 MB 90.6 us, 94.0 with them, of 64 MB 26.4 and 27.2, of 16 MB 10.2 and 10.5, normal-
// distributed values of 16 MB 9.8 and 10.0); in the steps of a collective they gain nothing and cost nothing there.
// Rows lie 20 words apart, so that eight neighbouring ones have no banks in common and a row's four loads are one address.
// Sums have a second set of rows, kOutlierRows further on, for outlier blocks: whatever such a block's planes hold for element 0 does
// not count (four streams of 256 MB 139.1 us without them, 139.8 with, 140.9 where every block chooses its set, not the outlier ones
// alone; from 17 to 21 rows apart they take the same).
constexpr int kMaskRows = 17, kOutlierRows = 17, kSumMaskRows = kOutlierRows + kMaskRows, kMaskPitch = 20;
template <int ROWS>
__device__ __forceinline__ void fill_masks(uint32_t* masks) {
  for (uint32_t i = threadIdx.x; i < 4u * ROWS; i += blockDim.x) {
    const int row = (int)(i >> 2), j = 4 * (int)(i & 3u);
    const int F = row < kOutlierRows ? row : row - kOutlierRows;
    const uint32_t all = row < kOutlierRows ? 0xffffffffu : ~kFirst;
    *reinterpret_cast<uint4*>(masks + kMaskPitch * row + j) =
        make_uint4(F > j ? all : 0u, F > j + 1 ? all : 0u, F > j + 2 ? all : 0u, F > j + 3 ? all : 0u);
  }
}
// (t & m) ^ s
__device__ __forceinline__ uint32_t and_xor(uint32_t t, uint32_t m, uint32_t s) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(d) : "r"(t), "r"(m), "r"(s));
  return d;
}
// four masks of the row at `row`, from plane 4 C on
template <int C>
__device__ __forceinline__ void four_masks(uint32_t row, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4 + %5];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(row), "n"(16 * C) : "memory");
}
__device__ __forceinline__ uint32_t mask_row(const uint32_t* masks, uint32_t row) { return smem_u32(masks) + 4u * kMaskPitch * row; }

// ---- stream -> block --------------------------------------------------------------------------------
// Reads the payload of the block with rate byte `rate` at byte `pos` of a staged stream: planes into T[0..W-1]
// (zero at and above F), the sign map in the planes' bit order, |d0| of an outlier block (else 0).  Every
// word is rebuilt from two neighbours by a funnel shift, whatever the block's alignment: with outlier blocks
// about, the lanes of a warp have all four alignments, and a second path for aligned blocks ran on top.
// Blocks without payload give zeros; up to 4 W + 8 bytes behind the payload are read (and ignored).
template <int W, int MASKED>
__device__ __forceinline__ void read_planes(const uint8_t* buf, const uint32_t* masks, uint32_t pos, uint32_t rate, bool any_outlier,
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
  sign = __funnelshift_r(word[0], word[1], sh);
  constexpr bool kMasks = W <= MASKED;
  uint32_t m[16];
  if (kMasks) {
    const uint32_t row = mask_row(masks, F);  // (F <= W)
    if (W > 0) four_masks<0>(row, m[0], m[1], m[2], m[3]);
    if (W > 4) four_masks<1>(row, m[4], m[5], m[6], m[7]);
    if (W > 8) four_masks<2>(row, m[8], m[9], m[10], m[11]);
    if (W > 12) four_masks<3>(row, m[12], m[13], m[14], m[15]);
  }
#pragma unroll
  for (int j = 1; j <= W; ++j) {
    const uint32_t x = __funnelshift_r(word[j], word[j + 1], sh);
    T[j - 1] = kMasks ? x & m[(j - 1) & 15] : (uint32_t)j <= F ? x : 0u;
  }
}

// sign map in the order of the stream's words <-> element i at bit 31 - i
__device__ __forceinline__ uint32_t swap_order(uint32_t sign) { return __byte_perm(sign, 0, 0x0123); }

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

// staged payload -> rows, sign map with element i at bit 31 - i; W (plane_width of the largest F of the warp) is warp-uniform.  The widths that data at the usual error
// bounds has come first and in line, so that the loop's instructions lie together (as a switch, with the longest
// variants in between: add of 64 MB 41.7 us, 40.3 this way; decode of 64 MB 22.4, 21.6)
// MASKED: widest blocks that are read with masks (see fill_masks)
template <int MASKED>
__device__ __forceinline__ void decode_rows(const uint8_t* buf, const uint32_t* masks, uint32_t pos, uint32_t rate, int W, uint32_t& sign,
                                            uint32_t& a0, uint32_t (&T)[32]) {
  const bool outl = __any_sync(0xffffffffu, rate & 0x80u);
  if (__builtin_expect(W == 12, 1)) { read_planes<12, MASKED>(buf, masks, pos, rate, outl, sign, a0, T); rows_of_block<12>(T, rate, a0); }
  else if (__builtin_expect(W == 8, 1)) { read_planes<8, MASKED>(buf, masks, pos, rate, outl, sign, a0, T); rows_of_block<8>(T, rate, a0); }
  else if (__builtin_expect(W == 16, 1)) { read_planes<16, MASKED>(buf, masks, pos, rate, outl, sign, a0, T); rows_of_block<16>(T, rate, a0); }
  else if (W == 4) { read_planes<4, MASKED>(buf, masks, pos, rate, outl, sign, a0, T); rows_of_block<4>(T, rate, a0); }
  else if (__builtin_expect(W == 0, 0)) { read_planes<0, MASKED>(buf, masks, pos, rate, outl, sign, a0, T); rows_of_block<0>(T, rate, a0); }
  else { read_planes<32, MASKED>(buf, masks, pos, rate, outl, sign, a0, T); rows_of_block<32>(T, rate, a0); }
  sign = swap_order(sign);
}

// 2^126 with the sign of element i: |d_i| * 2^-149 (the row as it stands, read as a float) times this is
// d_i * 2^-23, which fma accumulates exactly while the sum stays below 2^24 steps
__device__ __forceinline__ float sign_scale(uint32_t sign, int i) { return as_f(and_or(sign << i, kMsb, 0x7e800000u)); }
// |d_i| and sign -> d_i as a subnormal
__device__ __forceinline__ uint32_t signed_sub(uint32_t mag, uint32_t sign, int i) { return mag ^ ((sign << i) & kMsb); }


// ---- block -> stream --------------------------------------------------------------------------------
template <int MODE>
__host__ __device__ constexpr int lorenzo_stride() { return MODE == kModeVec ? 4 : 1; }

struct BlockCode {
  uint32_t rate;  // rate byte
  uint32_t len;   // payload bytes
  uint32_t nout;  // outlier bytes (0: plain layout)
  uint32_t a0;    // |d_0|
  uint32_t sign;  // sign map in the order of the stream's words
};

// values (float bits) -> deltas of the quantised values as subnormals, in place
template <int MODE>
__device__ __forceinline__ void deltas_sub(uint32_t (&w)[32], float recip, float one) {
  constexpr int S = lorenzo_stride<MODE>();
  const uint64_t recip2 = twice(recip), one2 = twice(one);
#pragma unroll
  for (int i = 0; i < 32; i += 2) quantise_sub2(w[i], w[i + 1], recip2, one2);
#pragma unroll
  for (int i = 31; i >= S; --i) w[i] = as_u(__fsub_rn(as_f(w[i]), as_f(w[i - S])));
}
// the same in int32
template <int MODE>
__device__ __forceinline__ void deltas_int(uint32_t (&w)[32], float recip) {
  constexpr int S = lorenzo_stride<MODE>();
#pragma unroll
  for (int i = 0; i < 32; ++i) w[i] = (uint32_t)quantise(as_f(w[i]), recip);
#pragma unroll
  for (int i = 31; i >= S; --i) w[i] -= w[i - S];
}
// a whole number held as a subnormal -> int32
__device__ __forceinline__ uint32_t sub_to_int(uint32_t bits) {
  const uint32_t m = (uint32_t)((int32_t)bits >> 31);
  return ((bits & 0x7fffffffu) ^ m) - m;
}
// int32 -> sign and magnitude, 31 bits (INT_MIN folds to -0, whose sign the stream keeps)
__device__ __forceinline__ uint32_t sign_magnitude(uint32_t d) { return ((uint32_t)abs((int32_t)d) & 0x7fffffffu) | (d & kMsb); }

// OR of the magnitudes of d_1 .. d_31
__device__ __forceinline__ uint32_t or_tail_of(const uint32_t (&d)[32]) {
  uint32_t o = d[31];
#pragma unroll
  for (int i = 1; i < 31; i += 2) o |= d[i] | d[i + 1];  // one 3-input operation per pair
  return o & 0x7fffffffu;
}
// the same of the rows of a decoded block (T[i ^ 7] = |d_i|)
__device__ __forceinline__ uint32_t or_rows_tail(const uint32_t (&T)[32]) {
  uint32_t o = 0;
#pragma unroll
  for (int i = 1; i < 32; ++i) o |= T[i ^ 7];
  return o;
}
// sign bits of the rows -> sign map in the order of the stream's words
__device__ __forceinline__ uint32_t signs_of(const uint32_t (&d)[32]) {
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < 32; ++i) s = __funnelshift_l(d[i], s, 1);
  return swap_order(s);
}
// rate byte and length of a block with |d_0| = c.a0 and magnitudes of f bits behind it:
// choose_rate() and payload_len() in fewer operations.  With f and w the bit widths of or_tail and |d_0| and o the
// bytes that w bits take, the plain layout has 4 + 4 max(f, w) bytes (none if that maximum is 0), the outlier layout
// 4 + 4 f + o, and the smaller one is taken, plain if equal.  For w <= f that is plain; for w > f it is the outlier layout if
// 4 w > 4 f + o, which w <= f never meets.
template <int MODE>
__device__ __forceinline__ void choose_code(BlockCode& c, uint32_t f) {
  const uint32_t w = 32u - (uint32_t)__clz((int)c.a0), o = (w + 7u) >> 3;
  const uint32_t top = f > w ? f : w;
  c.rate = top;
  c.len = top ? 4u * top + 4u : 0u;
  c.nout = 0;
  if (MODE != kModePlain && 4u * w > 4u * f + o) {
    c.rate = f + 32u * o + 96u;  // 0x80 | (o - 1) << 5 | f
    c.len = 4u * f + 4u + o;
    c.nout = o;
  }
}
// sign-magnitude deltas -> the block's code; d_0 of an outlier block is taken out of the planes
template <int MODE>
__device__ __forceinline__ BlockCode code_of(uint32_t (&d)[32], uint32_t or_tail) {
  BlockCode c;
  c.sign = signs_of(d);
  c.a0 = d[0] & 0x7fffffffu;
  choose_code<MODE>(c, 32u - (uint32_t)__clz((int)or_tail));
  if (c.nout) d[0] = 0;
  return c;
}

// Packs one block per lane into the ring at `base` (shared address, 16-byte aligned), the lane's payload at byte `rel`:
// outlier bytes, sign map, planes T[0..W-1] (those at and above F are zero).  Only whole words are stored.  The
// word in which a block starts is shared with the block before it: every lane first stores all its words behind
// that one, the last of them padded with zeros, then merges its first bytes into what the lane in front left.
// The ring must have 4 bytes behind the warp's payload.
template <int W>
__device__ __forceinline__ void pack_block(uint32_t base, uint32_t rel, const BlockCode& c, const uint32_t (&T)[32]) {
  const uint32_t F = c.rate & 31u;
  const uint32_t a0 = c.nout ? c.a0 : 0u;
  const uint32_t p2 = rel + c.nout;
  const uint32_t s0 = 8u * rel, s = 8u * p2;  // (funnel shifts take them modulo 32)
  const uint32_t first = base + (rel & ~3u), at = base + (p2 & ~3u);  // words of the first byte, of the sign map
  const uint32_t sign = c.sign;
  uint32_t head = __funnelshift_l(0u, a0, s0);
  if (c.len) {
    // words 1 .. F + 1 hold payload; as bits of a register seven comparisons turn into one instruction
    const uint32_t live = (4u << F) - 1u;
    uint32_t prev = sign;
#pragma unroll
    for (int j = 1; j <= W + 1; ++j) {
      const uint32_t next = j <= W ? T[j - 1] : 0u;
      const uint32_t v = __funnelshift_l(prev, next, s);
      if (W <= 16 ? (live & (1u << (j & 31))) != 0 : (uint32_t)j <= F + 1u) sts32(at + 4 * j, v);
      prev = next;
    }
    const uint32_t x = __funnelshift_l(0u, sign, s);
    if (at == first) head |= x;
    else sts32(at, __funnelshift_l(a0, 0u, s0) | x);
  }
  __syncwarp();
  if (c.len) sts32(first, (rel ? lds32(first) : 0u) | head);
  __syncwarp();
}
template <int W>
__device__ __forceinline__ void pack_w(uint32_t base, uint32_t rel, const BlockCode& c, const uint32_t (&d)[32]) {
  uint32_t T[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) T[i ^ 7] = W == 32 ? d[i] & 0x7fffffffu : d[i];  // (W <= 16: the sign bits drop out)
  if (W) planes_from_rows<W ? W : 4>(T);
  pack_block<W>(base, rel, c, T);
}
// W: plane_width of the largest F of the warp
__device__ __forceinline__ void pack_blocks(uint32_t base, uint32_t rel, const BlockCode& c, const uint32_t (&d)[32], int W) {
  if (__builtin_expect(W == 12, 1)) pack_w<12>(base, rel, c, d);
  else if (__builtin_expect(W == 8, 1)) pack_w<8>(base, rel, c, d);
  else if (__builtin_expect(W == 16, 1)) pack_w<16>(base, rel, c, d);
  else if (W == 4) pack_w<4>(base, rel, c, d);
  else if (__builtin_expect(W == 0, 0)) pack_w<0>(base, rel, c, d);
  else pack_w<32>(base, rel, c, d);
}

// ---- blocks as planes --------------------------------------------------------------------------------
// Sum of the contributions to one block as two's complement planes (hc_bitplane.h): kNarrow of them while `bound`, which no
// magnitude of the warp exceeds, fits them, else all 32, which wrap like an int32.
// |d_0| of outlier blocks, and a local d_0 that does not fit the planes of its warp, are summed apart.
// What bounds an add of streams is its instructions, at 15 warps an SM, and the latency of each warp's own chain.  A sub-tile of
// stream + stream takes 1299 warp instructions this way, 1605 by way of rows (gradients; 1478 and 1870 for a random walk), one of seven
// streams and fp32 3550 and 4380: 16 MB of a random walk 23.8 -> 20.3 us, 64 MB of gradients 49.2 -> 44.5, seven streams of 8 MB and
// their decode 25.1 -> 23.0.  With ONE stream and fp32 as many instructions are left (the rows of the local operand are there
// already) and their chain is longer: 64 MB 38.4 us by way of rows, 40.5 this way.
// A stream of 17 or 18 planes, which twenty would hold, is read in the wide code, for the masks of a block end at 16 (64 MB of blocks of
// 16, 17, 18 and 19 planes added 49.2, 53.8, 54.9 and 57.3 us; by way of rows 63.7, 72.9, 75.9 and 78.9); blocks of up to 4 planes are
// read like those of 8 (a smooth field of 64 MB 38.6 us; by way of rows, with code of their own width, 40.8).
// Two pieces of code, narrow and wide, not one for each width (44.0 us where this takes 44.5, but 21.6 against 20.3 for the random walk
// and 44.2 against 37.7 for three of them), and not groups of four planes as far as they are needed (46.4).
constexpr int kNarrow = 20;
struct PlaneSum {
  uint32_t A[32];
  uint32_t apart, bound;
};
__device__ __forceinline__ bool sum_wide(const PlaneSum& s) { return __any_sync(0xffffffffu, s.bound >> (kNarrow - 1)); }
__device__ __forceinline__ void sum_clear(PlaneSum& s) {
#pragma unroll
  for (int j = 0; j < kNarrow; ++j) s.A[j] = 0;
  s.apart = s.bound = 0;
}
// planes 8 B .. 8 B + 7 of a block (zero at and above F), exclusive or sign; word: the one that plane 8 B begins in; row: its masks
template <int B>
__device__ __forceinline__ void read_eight(uint32_t wp, uint32_t sh, uint32_t F, uint32_t row, uint32_t sign, uint32_t& word, uint32_t (&X)[32]) {
  uint32_t w[8], m[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = lds32(wp + 4 * (8 * B + 2 + j));
  if (B < 2) {
    four_masks<2 * B>(row, m[0], m[1], m[2], m[3]);
    four_masks<2 * B + 1>(row, m[4], m[5], m[6], m[7]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t x = __funnelshift_r(j ? w[j - 1] : word, w[j], sh);
    X[8 * B + j] = B < 2 ? and_xor(x, m[j], sign) : ((uint32_t)(8 * B + j) < F ? x : 0u) ^ sign;
  }
  word = w[7];
}
// Adds the staged payload at byte `pos` of buf; masks: see fill_masks.  However short it is, the 10 words from its sign map on are read,
// 18 if a block of the warp has more than 8 planes, 34 with more than 16: kSumReads bytes from `pos` on at most.  As everywhere, d_0 of an outlier block is the 31 bits of its bytes,
// and nothing of what its planes may hold for element 0 (an encoder that does not mask |INT_MIN|, a damaged stream).
constexpr int kSumReads = 4 + 4 * 34;  // bytes of d_0, words from the sign map on
__device__ __forceinline__ void sum_add(PlaneSum& s, const uint8_t* buf, const uint32_t* masks, uint32_t pos, uint32_t rate) {
  const uint32_t F = rate & 31u, W = __reduce_max_sync(0xffffffffu, F);
  uint32_t p2 = pos, a0 = 0, row = mask_row(masks, F < 16u ? F : 16u);
  if (__any_sync(0xffffffffu, rate & 0x80u)) {
    if (rate & 0x80u) {
      const uint32_t nout = ((rate >> 5) & 3u) + 1u;
      const uint32_t wa = smem_u32(buf) + (pos & ~3u);
      a0 = __funnelshift_r(lds32(wa), lds32(wa + 4u), 8u * (pos & 3u)) & (0xffffffffu >> (32u - 8u * nout)) & 0x7fffffffu;
      p2 += nout;
      row += 4u * kMaskPitch * kOutlierRows;
    }
  }
  const uint32_t sh = 8u * (p2 & 3u), wp = smem_u32(buf) + (p2 & ~3u);
  uint32_t X[32], word0 = lds32(wp), word = lds32(wp + 4u);
  const uint32_t sign = __funnelshift_r(word0, word, sh);
  read_eight<0>(wp, sh, F, row, sign, word, X);
  if (W > 8u) {
    read_eight<1>(wp, sh, F, row, sign, word, X);
  } else {
#pragma unroll
    for (int j = 8; j < 16; ++j) X[j] = sign;
  }
  s.apart += sign & kFirst ? 0u - a0 : a0;
  const bool was_wide = sum_wide(s);
  s.bound = W > 16u ? 0x7fffffffu : min(s.bound + (1u << W), 0x7fffffffu);
  if (__builtin_expect(sum_wide(s), 0)) {
    if (!was_wide) {
#pragma unroll
      for (int j = kNarrow; j < 32; ++j) s.A[j] = s.A[kNarrow - 1];
    }
    if (W > 16u) {
      read_eight<2>(wp, sh, F, row, sign, word, X);
      read_eight<3>(wp, sh, F, row, sign, word, X);
      if (rate & 0x80u) {  // (what the masks do for the planes below; as a mask of read_eight it cost the blocks without such planes 2 us of 140)
#pragma unroll
        for (int j = 16; j < 32; ++j) X[j] = bit_select(X[j], sign, ~kFirst);
      }
    } else {
#pragma unroll
      for (int j = 16; j < 32; ++j) X[j] = sign;
    }
    add_planes<32, 32>(s.A, X, sign);
  } else {
    add_planes<16, kNarrow>(s.A, X, sign);
  }
}
// Sum -> values (float bits).  In planes the sum of k streams costs k additions and one transposition.  The rows come out with B
// added to each (the top plane flipped), which makes them unsigned: their prefix sum is 32 fma, and what it has too much, a
// whole number of B, comes off by an addition on the same pipe, where signs would take a shift and a logic operation a value.
// Widths: 12 planes for sums of up to 11 bits, 16 for up to 15; the rest, with 32, goes by way of int32 (four streams of a random
// walk of 16 MB 25.1 us by way of a row for every stream, 20.4 this way).
template <int W>
__device__ __forceinline__ void biased_values(PlaneSum& s, float scale, uint32_t (&w)[32]) {
  constexpr int B = 1 << (W - 1);
  s.A[W - 1] = ~s.A[W - 1];
  rows_from_planes<W>(s.A);
  float q[32];
  const float apart = __fmul_rn((float)(int32_t)s.apart, 0x1p-23f);
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    q[i] = __fmaf_rn(as_f(s.A[i ^ 7]), 0x1p126f, i ? q[i - 1] : apart);
    w[i] = as_u(__fmul_rn(__fadd_rn(q[i], -0x1p-23f * (float)((i + 1) * B)), scale));
  }
}
// (stride-1 predictor only: no sum of streams of mode vec is decoded)
__device__ __forceinline__ void sum_values(PlaneSum& s, float scale, float eb, uint32_t (&w)[32]) {
  // no sum of a row leaves 24 bits: 32 magnitudes of 15 bits and B for each, and |d_0|'s part that is apart
  const bool exact = scale != 0.0f && s.bound <= 1u << 15 && s.apart + (1u << 22) < (1u << 23);
  if (__builtin_expect(__all_sync(0xffffffffu, exact), 1)) {
    if (__builtin_expect(__all_sync(0xffffffffu, s.bound <= 1u << 11), 1)) biased_values<12>(s, scale, w);
    else biased_values<16>(s, scale, w);
    return;
  }
  if (!sum_wide(s)) {
#pragma unroll
    for (int j = kNarrow; j < 32; ++j) s.A[j] = s.A[kNarrow - 1];
  }
  rows_from_planes<32>(s.A);
  uint32_t q[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    q[i] = s.A[i ^ 7] + (i ? q[i - 1] : s.apart);
    w[i] = as_u(__fmul_rn(__fmul_rn((float)(int32_t)q[i], eb), 2.0f));
  }
}
// Starts a sum with the block's own deltas: subnormals, or int32 (`ints`); or_tail: of the subnormals.
__device__ __forceinline__ void sum_local(PlaneSum& s, uint32_t (&d)[32], uint32_t or_tail, bool ints) {
  const uint32_t W = ints ? 32u : __reduce_max_sync(0xffffffffu, 32u - (uint32_t)__clz((int)or_tail));
  uint32_t (&A)[32] = s.A;
  s.apart = 0;
  if (__builtin_expect(W <= 16u, 1)) {
    if ((d[0] & 0x7fffffffu) >> W) {
      s.apart = sub_to_int(d[0]);
      d[0] = 0;
    }
    const uint32_t sign = signs_of(d);
#pragma unroll
    for (int i = 0; i < 32; ++i) A[i ^ 7] = d[i];
    planes_up_to_16(A, W);
    if (W <= 8u) {
#pragma unroll
      for (int j = 8; j < 16; ++j) A[j] = 0;
    } else if (W <= 12u) {
#pragma unroll
      for (int j = 12; j < 16; ++j) A[j] = 0;
    }
    uint32_t c = sign;
    negate_planes<16>(A, sign, c);
#pragma unroll
    for (int j = 16; j < kNarrow; ++j) A[j] = sign & ~c;
    s.bound = 1u << W;
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) A[i ^ 7] = ints ? d[i] : sub_to_int(d[i]);
    planes_from_rows<32>(A);
    s.bound = 0x7fffffffu;
  }
}
// Sum -> magnitude planes in A (zero at and above the planes of the block) and the block's code.
template <int MODE>
__device__ __forceinline__ BlockCode sum_code(PlaneSum& s) {
  BlockCode c;
  uint32_t (&A)[32] = s.A;
  const bool wide = sum_wide(s);
  c.sign = wide ? A[31] : A[kNarrow - 1];
  // magnitudes, how many planes they take without d_0, and |d_0|
  uint32_t carry = c.sign, f = 0, v = 0;
  negate_planes<kNarrow>(A, c.sign, carry);
  auto look = [&](int g) {
#pragma unroll
    for (int j = 4 * g; j < 4 * g + 4; ++j)
      if (A[j] & ~kFirst) f = j + 1;
    v |= firsts_of(A[4 * g], A[4 * g + 1], A[4 * g + 2], A[4 * g + 3]) >> 28 << 4 * g;
  };
#pragma unroll
  for (int g = 0; g < kNarrow / 4; ++g) look(g);
  if (__builtin_expect(wide, 0)) {
#pragma unroll
    for (int j = kNarrow; j < 31; ++j) {
      const uint32_t a = A[j];
      A[j] = xor3(a, c.sign, carry);
      carry &= a ^ c.sign;
    }
    A[31] = 0;  // 31 bits
#pragma unroll
    for (int g = kNarrow / 4; g < 8; ++g) look(g);
  } else {
#pragma unroll
    for (int j = kNarrow; j < 32; ++j) A[j] = 0;
  }
  if (c.sign & kFirst) v = v ? 0u - v : kMsb;  // (a sign without a magnitude: the smallest of the 32-bit integers)
  v += s.apart;
  c.sign = bit_select(c.sign, v >> 24, ~kFirst);
  c.a0 = (uint32_t)abs((int32_t)v) & 0x7fffffffu;
  choose_code<MODE>(c, f);
  // d_0 in the planes: as it came out of them where the block is a plain one, unless some of it was apart
  if (__any_sync(0xffffffffu, c.nout | s.apart)) {
    const uint32_t a0 = c.nout ? 0u : c.a0;
#pragma unroll
    for (int j = 0; j < 31; ++j) A[j] = bit_select(A[j], j <= 7 ? a0 << (7 - j) : a0 >> (j - 7), ~kFirst);
  }
  return c;
}
// packs the planes of a block per lane (see pack_block); W: plane_width of the largest F of the warp
__device__ __forceinline__ void pack_planes(uint32_t base, uint32_t rel, const BlockCode& c, const uint32_t (&A)[32], int W) {
  if (__builtin_expect(W == 12, 1)) pack_block<12>(base, rel, c, A);
  else if (__builtin_expect(W == 8, 1)) pack_block<8>(base, rel, c, A);
  else if (__builtin_expect(W == 16, 1)) pack_block<16>(base, rel, c, A);
  else if (W == 4) pack_block<4>(base, rel, c, A);
  else if (__builtin_expect(W == 0, 0)) pack_block<0>(base, rel, c, A);
  else pack_block<32>(base, rel, c, A);
}

// 16-byte units of copy_ring: source bytes start K words and sh bits into 16-byte aligned shared memory.  Not unrolled: a
// payload is one to three turns, and the four copies of an unrolled loop with its remainder cost more instructions and
// registers than they save (vec mode 40 MB: 19.0 us unrolled, 18.0 by two, 17.0 this way)
template <int K>
__device__ __forceinline__ void copy_units(uint32_t src, uint8_t* out, uint32_t units, uint32_t sh) {
#pragma unroll 1
  for (uint32_t u = threadIdx.x & 31u; u < units; u += 32u) {
    uint32_t a[8];
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(src + 16u * u) : "memory");
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]) : "r"(src + 16u * u + 16u) : "memory");
    *reinterpret_cast<uint4*>(out + 16u * u) =
        make_uint4(__funnelshift_r(a[K], a[K + 1], sh), __funnelshift_r(a[K + 1], a[K + 2], sh),
                   __funnelshift_r(a[K + 2], a[K + 3], sh), __funnelshift_r(a[K + 3], a[K + 4], sh));
  }
}
// Moves the `tot` bytes at ring address `src` (16-byte aligned) to `dst` in global memory, one warp: 16-byte stores
// for whole units, the bytes of the first and last partial unit one per lane.  The shift between the alignments of
// source and destination is the same for every unit: whole words by choosing registers, the rest by funnel shifts.
// Reads up to 16 bytes behind the payload.
__device__ __forceinline__ void copy_ring(uint32_t src, uint8_t* dst, uint32_t tot) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t head = (16u - ((uint32_t)reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u;
  if (head > tot) head = tot;
  const uint32_t units = (tot - head) >> 4, tail = (tot - head) & 15u;
  if (lane < 16u ? lane < head : lane - 16u < tail) {
    const uint32_t at = lane < 16u ? lane : head + 16u * units + lane - 16u;
    uint32_t b;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(b) : "r"(src + at) : "memory");
    dst[at] = (uint8_t)b;
  }
  switch (head >> 2) {
    case 0: copy_units<0>(src, dst + head, units, 8u * (head & 3u)); break;
    case 1: copy_units<1>(src, dst + head, units, 8u * (head & 3u)); break;
    case 2: copy_units<2>(src, dst + head, units, 8u * (head & 3u)); break;
    default: copy_units<3>(src, dst + head, units, 8u * (head & 3u)); break;
  }
}

}  // namespace dev
}  // namespace hc
