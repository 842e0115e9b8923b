// Cells as seven signed base-256 digits, and where their planes lie (see cla_split.cu).
#pragma once
#include <stdint.h>

namespace cla {

constexpr int SP_DIG = 7;
constexpr int SP_COLS = 128;              // columns of a block
constexpr int SP_PLANE = SP_COLS * 16;    // bytes of a digit of 16 rows
constexpr int SP_HALF = SP_DIG * SP_PLANE;  // all digits of 16 rows

__device__ __forceinline__ double split_scale(int e) { return scalbn(1.0, 55 - e); }
// The digits of x, |x| <= 0.99 * 2^e, the last one in byte 0. GUARD: what the guard multiplies in their place, digit 0 whether the
// cell differs from zero (the cell itself, not its digits) and digit 1 its magnitude's leading seven bits, rounded down; bad: a value
// that has no digits (not finite, or beyond the bound).
template <bool GUARD>
__device__ __forceinline__ unsigned long long split_pack(double x, double scale, bool& bad) {
  const double y = x * scale;
  if (GUARD) {
    bad |= !(fabs(y) <= 0x1p55);
    return (unsigned long long)(x != 0.0) << 48 | (unsigned long long)min((int)(fabs(y) * 0x1p-48), 126) << 40;
  }
  // + 128 in every byte makes the bytes the digits + 128
  return ((unsigned long long)__double2ll_rn(y) + 0x80808080808080ull) ^ 0x80808080808080ull;
}
// Byte i of four words to word i of the result
__device__ __forceinline__ void transpose4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&o)[4]) {
  const uint32_t ab = __byte_perm(a, b, 0x5140), cd = __byte_perm(c, d, 0x5140);
  const uint32_t AB = __byte_perm(a, b, 0x7362), CD = __byte_perm(c, d, 0x7362);
  o[0] = __byte_perm(ab, cd, 0x5410);
  o[1] = __byte_perm(ab, cd, 0x7632);
  o[2] = __byte_perm(AB, CD, 0x5410);
  o[3] = __byte_perm(AB, CD, 0x7632);
}
// 16 rows of column c to their place: p points at the 16 rows' first plane of the column's block
template <bool GUARD>
__device__ __forceinline__ void split_store(uint8_t* p, int c, const unsigned long long (&v)[16]) {
  uint32_t w[SP_DIG][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t o[4];
    transpose4((uint32_t)v[4 * q], (uint32_t)v[4 * q + 1], (uint32_t)v[4 * q + 2], (uint32_t)v[4 * q + 3], o);
#pragma unroll
    for (int i = 0; i < 4; i++) w[6 - i][q] = o[i];
    transpose4((uint32_t)(v[4 * q] >> 32), (uint32_t)(v[4 * q + 1] >> 32), (uint32_t)(v[4 * q + 2] >> 32), (uint32_t)(v[4 * q + 3] >> 32), o);
#pragma unroll
    for (int i = 0; i < 3; i++) w[2 - i][q] = o[i];
  }
  p += (c % SP_COLS) * 16;
#pragma unroll
  for (int d = 0; d < (GUARD ? 2 : SP_DIG); d++) *(uint4*)(p + (size_t)d * SP_PLANE) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
}

}  // namespace cla
