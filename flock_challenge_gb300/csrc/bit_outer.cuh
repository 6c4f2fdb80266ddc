// Sums of products sum_j a_j b_j in GF(2^128) on the tensor cores.
//
// The product is bilinear over GF(2): sum_j a_j b_j = sum_{p, q} x^(p + q)
// parity(#{j : bit p of a_j and bit q of b_j}), so the sum over any number of
// pairs is one 128 x 128 matrix of counts, the summed index running over the
// pairs (tc.cuh), and the reduction to a field element is paid once. Per pair
// and product this is two operands of 64 bytes (a bit per nibble) written to
// shared memory and read by the MMAs, and 72 logic operations, against about
// 400 instructions of a carry-less product.
//
// Both sums of a round's message, over a_1 b_1 (or a_0 b_0) and (a_0 + a_1)
// (b_0 + b_1), are taken together. A warp holds 128 pairs of one factor, lane
// l value l & 1 (the plain one on one lane, the sum on the other) of the pairs
// 16 k + l / 2 (k < 8); a slot is one such warp tile of each factor. A tile of
// one sum is four planes of 32 pairs, a plane being [128 rows p][16 bytes]: the
// lane fills word (l / 2) & 3 of the rows of plane l / 8 with its eight pairs,
// one nibble each. Planes lie 16 bytes more than 2 KB apart, the two sums' tiles
// therefore 64 bytes off a multiple of 128, which puts the 32 lanes' stores on
// 32 banks.
#pragma once
#include "gf128.cuh"
#include "tc.cuh"

namespace bo {

constexpr int PLANE = 128 * 16 + 16, SUM = 4 * PLANE, SIDE = 2 * SUM, SLOT = 2 * SIDE;
constexpr int TILE = 128;  // pairs
static_assert(SUM % 128 == 64 && SUM % 16 == 0, "the two sums' tiles on different halves of the banks");

// Word w of the lane's eight values (u[k], k < 8) to rows 32 w .. 32 w + 31:
// an 8 x 8 transpose of nibbles, then the four masks. d: the lane's word of row
// 32 w. Rows 4 n + m stand for 0.5, 1, 2, 0.5 (m = 0..3) per set bit.
__device__ __forceinline__ void put_word(const uint32_t (&u)[8], uint32_t* d) {
  uint32_t lo[4], hi[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const uint32_t a = u[2 * c], b = u[2 * c + 1];
    lo[c] = (a & 0x0F0F0F0Fu) | ((b << 4) & 0xF0F0F0F0u);
    hi[c] = ((a >> 4) & 0x0F0F0F0Fu) | (b & 0xF0F0F0F0u);
  }
  auto bytes = [&](const uint32_t (&x)[4], int first) {
    const uint32_t l01 = __byte_perm(x[0], x[1], 0x5140), h01 = __byte_perm(x[0], x[1], 0x7362);
    const uint32_t l23 = __byte_perm(x[2], x[3], 0x5140), h23 = __byte_perm(x[2], x[3], 0x7362);
    const uint32_t t[4] = {__byte_perm(l01, l23, 0x5410), __byte_perm(l01, l23, 0x7632),
                           __byte_perm(h01, h23, 0x5410), __byte_perm(h01, h23, 0x7632)};
#pragma unroll
    for (int i = 0; i < 4; i++) {  // nibble 2 i + first of the values: bits 4 (2 i + first) ..
      uint32_t* r = d + 16 * (2 * i + first);
      r[0] = t[i] & 0x11111111u;
      r[4] = t[i] & 0x22222222u;
      r[8] = t[i] & 0x44444444u;
      r[12] = (t[i] >> 3) & 0x11111111u;
    }
  };
  bytes(lo, 0);
  bytes(hi, 1);
}

// The lane's eight values into its warp's operand tile, of sum `sum`.
__device__ __forceinline__ void put_tile(const gf128 (&v)[8], uint8_t* side, int sum) {
  const int lane = threadIdx.x & 31;
  uint32_t* d = reinterpret_cast<uint32_t*>(side + sum * SUM + (lane >> 3) * PLANE) + ((lane >> 1) & 3);
#pragma unroll
  for (int w = 0; w < 4; w++) {
    uint32_t u[8];
#pragma unroll
    for (int k = 0; k < 8; k++) u[k] = v[k].w[w];
    put_word(u, d + 128 * w);
  }
}

// The MMAs of one slot (factor a's tiles, then b's, at shared address s): sum i
// into the 128 columns at d + 128 i.
__device__ __forceinline__ void mma_slot(uint32_t s, uint32_t d, uint32_t sf, bool first) {
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const uint32_t a = s + i * SUM + 2 * q * PLANE;
      tc::mma_mxf4(d + 128 * i, tc::operand(a, PLANE, 128), tc::operand(a + SIDE, PLANE, 128), tc::mxf4_desc(128, 128),
                   sf, sf + 16, !first || q > 0);
    }
}

// The counts at column d of TMEM as field elements' parts: called by the four
// warps of a warpgroup-aligned set (warp & 3 = their quadrant of rows); the
// quadrant's 160-bit partial polynomial, times x^(32 quadrant), to out[5] by
// lane 0.
__device__ __forceinline__ void read_quadrant(uint32_t d, uint32_t* out) {
  const int lane = threadIdx.x & 31, quad = (threadIdx.x >> 5) & 3;
  // row p = 32 quad + lane stands for 0.5, 1, 2, 0.5: undone here, as the columns' below
  const float row = (lane & 3) == 1 ? 1.0f : (lane & 3) == 2 ? 0.5f : 2.0f;
  uint32_t m[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int w = 0; w < 4; w++) {
    uint32_t r[32];
    tc::tmem_load32(d + ((uint32_t)(32 * quad) << 16) + 32 * w, r);
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const float col = (j & 3) == 1 ? 1.0f : (j & 3) == 2 ? 0.5f : 2.0f;
      // counts below 2^23: the low mantissa bit is the parity
      const uint32_t par = __float_as_uint(fmaf(__uint_as_float(r[j]), row * col, 8388608.0f)) & 1u;
      m[w] |= par << j;
    }
  }
  // x^lane times the row's polynomial, summed over the quadrant's rows
  const uint32_t s[5] = {m[0] << lane, __funnelshift_l(m[0], m[1], lane), __funnelshift_l(m[1], m[2], lane),
                         __funnelshift_l(m[2], m[3], lane), __funnelshift_l(m[3], 0u, lane)};
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const uint32_t v = __reduce_xor_sync(0xffffffffu, s[k]);
    if (lane == 0) out[k] = v;
  }
}

// The four quadrants' parts as the field element.
__device__ __forceinline__ gf128 combine(const uint32_t (*q)[5]) {
  uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int i = 0; i < 5; i++)
      if (k + i < 8) w[k + i] ^= q[k][i];
  return gf_reduce(w[0] | ((uint64_t)w[1] << 32), w[2] | ((uint64_t)w[3] << 32), w[4] | ((uint64_t)w[5] << 32),
                   w[6] | ((uint64_t)w[7] << 32));
}

}  // namespace bo
