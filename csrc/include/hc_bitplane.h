// In-register bit-plane transposition for one 32-element block held by ONE thread.
//
// The stream stores a block's magnitudes as F bit planes: plane p is a big-endian 32-bit map in
// which element i sits at bit 31 - i.  Read as a little-endian machine word, element i therefore
// sits at bit (i ^ 7).  With rows A[j] = mag[j ^ 7] (a compile-time renaming of registers) the
// planes are exactly the 32x32 bit-matrix transpose:  T[p] bit j = A[j] bit p.
//
// The transpose is five independent stages (one per index bit); stage `s` swaps bit s of the row
// index with bit s of the column index.  Stages 16 and 8 are byte permutes (PRMT), stages 4, 2, 1
// are shift-xor swaps.  When every magnitude of the block fits W bits (W = 4, 8, 12, 16) the upper rows
// of the result are known zero and most of the network disappears, which is what makes the
// thread-per-block layout cheaper than one warp ballot per plane: 114 instructions a block at W = 12, 140 at W = 16 (150 and 188 before the
// bit selects were single instructions; isolated loops, counted), independent of F.
//
// The reference packs planes with 32 shift/or pairs per output byte (HomComp/src/GSZ.cu:1698-1735).
#pragma once
#include "hc_format.h"

namespace hc {

// byte permute; selector bit 3 gives the chosen byte's sign bit in all eight places (which __byte_perm leaves out)
HC_HD uint32_t perm(uint32_t a, uint32_t b, uint32_t sel) {
#if defined(__CUDA_ARCH__)
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
#else
  uint64_t v = ((uint64_t)b << 32) | a;
  uint32_t r = 0;
  for (int k = 0; k < 4; ++k) {
    uint32_t byte = (uint32_t)(v >> (8 * ((sel >> (4 * k)) & 7))) & 0xffu;
    if ((sel >> (4 * k)) & 8u) byte = byte & 0x80u ? 0xffu : 0u;
    r |= byte << (8 * k);
  }
  return r;
#endif
}

// bits of a where m has ones, of b where it has zeros.  One 3-input operation; written as plain C, two constant masks
// (m and ~m) each take an operation of their own, because an instruction holds one immediate
HC_HD uint32_t bit_select(uint32_t a, uint32_t b, uint32_t m) {
#if defined(__CUDA_ARCH__)
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xe4;" : "=r"(d) : "r"(a), "r"(b), "r"(m));
  return d;
#else
  return (a & m) | (b & ~m);
#endif
}

// swap the bits of A[k] selected by ~m with the bits of A[k + s] selected by m (m << s == ~m).  Written as two
// bit selects: two shifts and two 3-input logic operations a pair, one operation less than the xor-swap form
template <int S>
HC_HD void swap_stage(uint32_t& lo, uint32_t& hi) {
  constexpr uint32_t m = S == 4 ? 0x0f0f0f0fu : (S == 2 ? 0x33333333u : 0x55555555u);
  const uint32_t l = lo, h = hi;
  lo = bit_select(l, h << S, m);
  hi = bit_select(l >> S, h, m);
}

// Forward: rows A[0..31] hold values below 2^W; on return A[0..W-1] hold planes 0..W-1.
// Rows W..31 are unspecified afterwards.  For W <= 16 the bits of the rows at and above 16 are ignored
// (stage 16 picks the low halves).
template <int W>
HC_HD void planes_from_rows(uint32_t (&A)[32]) {
  static_assert(W == 4 || W == 8 || W == 12 || W == 16 || W == 32, "W");
  // stage 16
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    uint32_t lo = A[k], hi = A[k + 16];
    A[k] = perm(lo, hi, 0x5410);
    if (W > 16) A[k + 16] = perm(lo, hi, 0x7632);
  }
  // stage 8
#pragma unroll
  for (int h = 0; h < (W > 16 ? 32 : 16); h += 16) {
#pragma unroll
    for (int k = h; k < h + 8; ++k) {
      uint32_t lo = A[k], hi = A[k + 8];
      A[k] = perm(lo, hi, 0x6240);
      if (W > 8) A[k + 8] = perm(lo, hi, 0x7351);
    }
  }
  constexpr int R = W == 12 ? 8 : W;  // rows with a full stage 4
  // stage 4
  if (W == 4) {
#pragma unroll
    for (int k = 0; k < 4; ++k) A[k] = bit_select(A[k], A[k + 4] << 4, 0x0f0f0f0fu);
  } else {
#pragma unroll
    for (int k = 0; k < R; ++k)
      if ((k & 4) == 0) swap_stage<4>(A[k], A[k + 4]);
    if (W == 12) {
#pragma unroll
      for (int k = 8; k < 12; ++k) A[k] = bit_select(A[k], A[k + 4] << 4, 0x0f0f0f0fu);
    }
  }
#pragma unroll
  for (int k = 0; k < W; ++k)
    if ((k & 2) == 0) swap_stage<2>(A[k], A[k + 2]);
#pragma unroll
  for (int k = 0; k < W; ++k)
    if ((k & 1) == 0) swap_stage<1>(A[k], A[k + 1]);
}

// The same for rows of W bits, W known at run time and from 0 to 16, in one piece of code for all of them: planes 0 .. 7, from W = 9 on
// 0 .. 11, from W = 13 on 0 .. 15.  What the entries behind them hold is not said.
HC_HD void planes_up_to_16(uint32_t (&A)[32], uint32_t W) {
#pragma unroll
  for (int k = 0; k < 16; ++k) A[k] = perm(A[k], A[k + 16], 0x5410);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t lo = A[k], hi = A[k + 8];
    A[k] = perm(lo, hi, 0x6240);
    A[k + 8] = perm(lo, hi, 0x7351);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) swap_stage<4>(A[k], A[k + 4]);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if ((k & 2) == 0) swap_stage<2>(A[k], A[k + 2]);
#pragma unroll
  for (int k = 0; k < 8; k += 2) swap_stage<1>(A[k], A[k + 1]);
  if (W <= 8) return;
  if (W <= 12) {
#pragma unroll
    for (int k = 8; k < 12; ++k) A[k] = bit_select(A[k], A[k + 4] << 4, 0x0f0f0f0fu);
  } else {
#pragma unroll
    for (int k = 8; k < 12; ++k) swap_stage<4>(A[k], A[k + 4]);
    swap_stage<2>(A[12], A[14]);
    swap_stage<2>(A[13], A[15]);
    swap_stage<1>(A[12], A[13]);
    swap_stage<1>(A[14], A[15]);
  }
  swap_stage<2>(A[8], A[10]);
  swap_stage<2>(A[9], A[11]);
  swap_stage<1>(A[8], A[9]);
  swap_stage<1>(A[10], A[11]);
}

// Inverse: A[0..W-1] hold planes 0..W-1 (planes >= F are zero); on return A[0..31] are the rows.
// Entries A[W..31] are ignored on input.
template <int W>
HC_HD void rows_from_planes(uint32_t (&A)[32]) {
  static_assert(W == 4 || W == 8 || W == 12 || W == 16 || W == 32, "W");
#pragma unroll
  for (int k = 0; k < W; ++k)
    if ((k & 1) == 0) swap_stage<1>(A[k], A[k + 1]);
#pragma unroll
  for (int k = 0; k < W; ++k)
    if ((k & 2) == 0) swap_stage<2>(A[k], A[k + 2]);
  constexpr int R = W == 12 ? 8 : W;  // rows with a full stage 4
  if (W == 4 || W == 12) {
#pragma unroll
    for (int k = W - 4; k < W; ++k) {
      uint32_t v = A[k];
      A[k] = v & 0x0f0f0f0fu;
      A[k + 4] = (v >> 4) & 0x0f0f0f0fu;
    }
  }
  if (W != 4) {
#pragma unroll
    for (int k = 0; k < R; ++k)
      if ((k & 4) == 0) swap_stage<4>(A[k], A[k + 4]);
  }
  if (W <= 8) {  // stages 8 and 16 at once: every byte of the eight registers is a row
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t v = A[k];
      A[k] = perm(v, 0u, 0x4440);
      A[k + 8] = perm(v, 0u, 0x4441);
      A[k + 16] = perm(v, 0u, 0x4442);
      A[k + 24] = perm(v, 0u, 0x4443);
    }
    return;
  }
  if (W == 12) {  // the same: two bytes a row, the upper one below 16, so that its sign (selectors 8 and up) fills the rest
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t lo = A[k], hi = A[k + 8];
      A[k] = perm(lo, hi, 0xcc40);
      A[k + 8] = perm(lo, hi, 0xdd51);
      A[k + 16] = perm(lo, hi, 0xee62);
      A[k + 24] = perm(lo, hi, 0xff73);
    }
    return;
  }
  // stage 8
#pragma unroll
  for (int h = 0; h < (W > 16 ? 32 : 16); h += 16) {
#pragma unroll
    for (int k = h; k < h + 8; ++k) {
      uint32_t lo = A[k], hi = A[k + 8];
      A[k] = perm(lo, hi, 0x6240);
      A[k + 8] = perm(lo, hi, 0x7351);
    }
  }
  // stage 16
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    uint32_t lo = A[k], hi = (W > 16) ? A[k + 16] : 0u;
    A[k] = perm(lo, hi, 0x5410);
    A[k + 16] = perm(lo, hi, 0x7632);
  }
}

// ---- sums in bit planes ---------------------------------------------------------------------------------
// A block's 32 integers as two's complement planes: A[p] holds bit p of every element, A[N - 1] the signs, in the bit order of
// the stream's words.  Adding a block of a stream, whose planes and sign map stand there already, takes three logic operations a
// plane; by way of rows it takes the transposition (114 operations at 12 planes) and three a row (96), and a result that goes back
// into a stream is transposed once more.
HC_HD uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0x96;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
#else
  return a ^ b ^ c;
#endif
}
HC_HD uint32_t majority(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xe8;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
#else
  return (a & b) | (c & (a | b));
#endif
}
// A += the integers with magnitude planes X[0 .. W-1] ^ sign and sign map `sign`, modulo 2^N
template <int W, int N>
HC_HD void add_planes(uint32_t (&A)[32], const uint32_t (&X)[32], uint32_t sign) {
  static_assert(W <= N && N <= 32, "planes");
  uint32_t c = sign;  // -m = ~m + 1
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t x = j < W ? X[j] : sign, a = A[j];
    A[j] = xor3(a, x, c);
    if (j + 1 < N) c = majority(a, x, c);
  }
}
// N planes (A ^ sign) + sign: magnitudes into two's complement, or back
template <int N>
HC_HD void negate_planes(uint32_t (&A)[32], uint32_t sign, uint32_t& c) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t a = A[j];
    A[j] = xor3(a, sign, c);
    c &= a ^ sign;
  }
}
// bit 7 of the words a0 .. a3 as bits 31 .. 28 (a3 .. a0), other bits below them
HC_HD uint32_t firsts_of(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
  const uint32_t v = perm(perm(a0, a1, 0x0040), perm(a2, a3, 0x0040), 0x5410) & 0x80808080u;
  return v * ((1u << 21) | (1u << 14) | (1u << 7) | 1u);
}

// smallest supported width that holds F planes (F in 0..31); 0 means "no planes at all"
HC_HD int plane_width(uint32_t F) {
  return F == 0 ? 0 : (F <= 4 ? 4 : (F <= 8 ? 8 : (F <= 12 ? 12 : (F <= 16 ? 16 : 32))));
}

}  // namespace hc
