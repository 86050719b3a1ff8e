// Digit slicing shared by the tensor-core GEMM kernels: the power-of-two
// row/column scale, the balanced signed digits of an FP64 value as exact 16-bit
// values (6 of 9 bits, FP16, in the tiled form; 7 of 7 bits, BF16, in the fused
// form), and the 128-byte swizzled K-major operand layout of tcgen05
// shared-memory descriptors.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

namespace tn {
namespace {

__device__ __forceinline__ uint32_t swz_off(int r, int c) {  // row r (0..), 16-byte chunk c (0..7)
  return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}

// power-of-two exponent e with |x| < 2^e for every x of a row/column whose
// largest magnitude has bit pattern maxbits (0 -> 0)
__device__ __forceinline__ int exp_of(uint64_t maxbits) {
  if (maxbits == 0) return 0;
  int ef = (int)(maxbits >> 52);
  if (ef == 0) return (63 - __clzll((long long)maxbits)) - 1073;  // subnormal: |x| < 2^(msb+1-1074)
  return ef - 1022;
}

// The FP32 bit pattern of x * 2^(7 - e), rounded to nearest even, the scaling
// done on the exponent field.  Integer operations: a cvt.f32.f64 runs on the
// FP64 pipe (two per clock and SM), which made the one-digit slices take longer
// than the six of the split form.
__device__ __forceinline__ uint32_t scaled_f32_bits(double x, int e) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int ef = (int)((hi >> 20) & 0x7FFu);
  const int fe = ef + 7 - e - 896;  // the FP32 exponent field
  if (ef != 0 && fe >= 1 && fe <= 254) {
    const uint32_t mant = ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    const uint32_t up = ((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (mant & 1u)) >> 29;
    return (hi & 0x80000000u) | (((uint32_t)fe << 23) + mant + up);
  }
  if (((hi << 1) | lo) == 0) return hi;               // zero of either sign
  return __float_as_uint((float)ldexp(x, 7 - e));     // subnormal or far below the row's scale
}

// ---------------------------------------------------------------- slicing
// 8 consecutive-k values of one row -> NS slices of 8 bf16 (packed in uint4).
//
// NS = 7: X = |x| * 2^(49 - e) rounded to the nearest integer (X <= 2^49),
// V = +-X, and the balanced base-128 digits of V (d_1..d_6 in [-64, 63],
// d_0 = the rest, |d_0| <= 129).  They are the plain base-128 digits of
// Y = V + 64 * (1 + 128 + ... + 128^5), each minus 64 (the representation is
// unique, so this equals peeling digits off from the bottom), read out of the
// two 32-bit halves of Y by shifts and masks.  d * 2^-7s is formed exactly in
// FP32 from the bit pattern of 1.5 * 2^(23-7s) + d * 2^-7s (integer add into
// the mantissa, one exact subtraction); it has at most 8 significant bits, so
// its BF16 pattern is the top half of the FP32 pattern.
// NS = 1 (fast mode): the BF16 rounding of the FP32 rounding of x * 2^(7-e),
// the scaling done on the exponent field.
template <int NS>
__device__ __forceinline__ void make_slices(const double (&x)[8], int e, uint4 (&out)[NS]) {
  static_assert(NS == 1 || NS == 7, "7 digits (split) or one BF16 slice (fast)");
  uint32_t packed[NS][4];
#pragma unroll
  for (int j = 0; j < 4; j++) {  // pair by pair, so few digits are held at once
    uint32_t hbits[NS][2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint64_t bits = (uint64_t)__double_as_longlong(x[2 * j + i]);
      const int ef = (int)((bits >> 52) & 0x7FF);
      if (NS == 1) {
        hbits[0][i] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(__uint_as_float(scaled_f32_bits(x[2 * j + i], e)))) << 16;
      } else {
        uint64_t mant = bits & ((1ull << 52) - 1);
        int E = -1022;
        if (ef) {
          mant |= 1ull << 52;
          E = ef - 1023;
        }
        const int sh = 3 + e - E;  // X = mant * 2^(E - 52) * 2^(49 - e)
        const uint64_t X = (sh >= 64) ? 0ull : (sh > 0 ? ((mant + (1ull << (sh - 1))) >> sh) : (mant << (-sh)));
        const long long V = (bits >> 63) ? -(long long)X : (long long)X;
        if constexpr (NS == 7) {
          const uint64_t Y = (uint64_t)(V + 2216338399296ll);  // + 64 * (128^6 - 1) / 127
          const uint32_t lo = (uint32_t)Y, hi = (uint32_t)(Y >> 32);
          int d[7];
          d[6] = (int)(lo & 127u) - 64;
          d[5] = (int)((lo >> 7) & 127u) - 64;
          d[4] = (int)((lo >> 14) & 127u) - 64;
          d[3] = (int)((lo >> 21) & 127u) - 64;
          d[2] = (int)(__funnelshift_r(lo, hi, 28) & 127u) - 64;
          d[1] = (int)((hi >> 3) & 127u) - 64;
          d[0] = (int)hi >> 10;
#pragma unroll
          for (int s = 0; s < 7; s++) {
            const float magic = __uint_as_float(0x4B400000u - ((uint32_t)(7 * s) << 23));  // 1.5 * 2^(23-7s)
            hbits[s][i] = __float_as_uint(__uint_as_float(__float_as_uint(magic) + (uint32_t)d[s]) - magic);
          }
        }
      }
    }
#pragma unroll
    for (int s = 0; s < NS; s++) packed[s][j] = __byte_perm(hbits[s][0], hbits[s][1], 0x7632);
  }
#pragma unroll
  for (int s = 0; s < NS; s++) out[s] = make_uint4(packed[s][0], packed[s][1], packed[s][2], packed[s][3]);
}

// The six digits of the tiled split form: V = x * 2^(53 - e) rounded to the
// nearest integer (|V| <= 2^53) and its balanced base-512 digits (d_1..d_5 in
// [-256, 255], |d_0| <= 256) as FP16 integers.  Y = 512 (V + 256 (1 + 512 + ...
// + 512^5)), below 2^64, has the digits plus 256 at bits 9, 18, 27, 36, 45 and
// 54; two elements' worth of one are packed into the mantissas of two FP16 in
// [1024, 2048) and 1280 subtracted.  About 30 integer instructions an element:
// the sign goes in as a bit inversion (V's last 2^-9), a shift past the top gives
// 0 for elements below 2^-62 of the scale and for zeros, and only where the
// scale itself is near the subnormals does an element's own exponent take the
// general form.  (The same in BF16, element by element with 64-bit shifts and a
// rounding of its own, took about 65; slicing 80000 x 400 153 -> 138 us.)
__device__ __forceinline__ void make_digits(const double (&x)[8], int e, uint4 (&out)[6]) {
  constexpr uint64_t kBias = (256ull * ((1ull << 54) - 1) / 511) * 512 + 256;  // and half a unit: rounds
  uint32_t lo[8], hi[8];
  if (e > -900) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t h = (uint32_t)__double2hiint(x[i]), l = (uint32_t)__double2loint(x[i]);
      const uint32_t m = (h & 0xFFFFFu) | 0x100000u, t1 = __funnelshift_l(l, m, 9), t0 = l << 9;  // mantissa * 512
      const int sh = min(e + 1022 - (int)((h >> 20) & 0x7FFu), 63);
      const bool far = sh >= 32;
      const uint32_t a1 = far ? 0u : t1, a0 = far ? t1 : t0, s = (uint32_t)((int)h >> 31);
      const uint64_t w = ((uint64_t)((a1 >> (sh & 31)) ^ s) << 32) | (__funnelshift_r(a0, a1, sh) ^ s);
      const uint64_t y = w + kBias;
      lo[i] = (uint32_t)y, hi[i] = (uint32_t)(y >> 32);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint64_t bits = (uint64_t)__double_as_longlong(x[i]);
      const int ef = (int)((bits >> 52) & 0x7FF);
      const uint64_t mant = (bits & ((1ull << 52) - 1)) | (ef ? 1ull << 52 : 0);
      const int sh = e + 1022 - max(ef, 1);  // V = mant * 2^-sh
      const uint64_t X = sh >= 64 ? 0ull : (sh > 0 ? (mant + (1ull << (sh - 1))) >> sh : mant << -sh);
      const uint64_t y = (((bits >> 63) ? 0ull - X : X) << 9) + kBias;
      lo[i] = (uint32_t)y, hi[i] = (uint32_t)(y >> 32);
    }
  }
  auto digit = [](uint32_t two, uint32_t mask) {
    const uint32_t v = (two & mask) | 0x64006400u;
    const __half2 d = __hsub2(*(const __half2*)&v, __half2(__ushort_as_half(0x6500), __ushort_as_half(0x6500)));
    return *(const uint32_t*)&d;
  };
  uint32_t packed[6][4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t l0 = lo[2 * j], l1 = lo[2 * j + 1], h0 = hi[2 * j], h1 = hi[2 * j + 1];
    packed[0][j] = digit(__byte_perm(h0, h1, 0x7632) >> 6, 0x03FF03FFu);  // bits 22..31 of the high words
    packed[1][j] = digit(__byte_perm(h0, h1, 0x6521) >> 5, 0x01FF01FFu);  // 13..21
    packed[2][j] = digit(__byte_perm(h0, h1, 0x5410) >> 4, 0x01FF01FFu);  // 4..12
    packed[3][j] = digit(__byte_perm(__funnelshift_r(l0, h0, 27), __funnelshift_r(l1, h1, 27), 0x5410), 0x01FF01FFu);
    packed[4][j] = digit(__byte_perm(l0, l1, 0x7632) >> 2, 0x01FF01FFu);  // 18..26 of the low words
    packed[5][j] = digit(__byte_perm(l0, l1, 0x6521) >> 1, 0x01FF01FFu);  // 9..17
  }
#pragma unroll
  for (int s = 0; s < 6; s++) out[s] = make_uint4(packed[s][0], packed[s][1], packed[s][2], packed[s][3]);
}

// TF32 fast mode: 8 consecutive-k values of one row as TF32 patterns of
// x * 2^(7 - e) (FP32 with the 13 low mantissa bits rounded off, to nearest,
// ties away from zero), packed as two 16-byte chunks.  The scaling is done on
// the exponent field as in the BF16 fast mode.
__device__ __forceinline__ void make_tf32(const double (&x)[8], int e, uint4 (&out)[2]) {
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t u = scaled_f32_bits(x[i], e);
    w[i] = ((u & 0x7F800000u) == 0x7F800000u) ? u : ((u + 0x1000u) & 0xFFFFE000u);
  }
  out[0] = make_uint4(w[0], w[1], w[2], w[3]);
  out[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// S * 2^q as the nearest double (ties to even), integer operations only (the
// FP64 units and FP64 conversions run at ~2 per clock per SM on GB300)
__device__ __forceinline__ double fixed_to_double(long long S, int q) {
  if (S == 0) return 0.0;
  const uint64_t sign = (uint64_t)S & (1ull << 63);
  uint64_t mag = S < 0 ? (uint64_t)(-S) : (uint64_t)S;
  const int lz = __clzll((long long)mag);
  mag <<= lz;                                        // leading one at bit 63
  const int E = 63 - lz + q;                         // value = mag * 2^(E - 63)
  const uint32_t rem = (uint32_t)mag & 0x7FFu;
  const uint64_t r = (mag >> 11) + (uint64_t)((rem > 0x400u) | ((rem == 0x400u) & (uint32_t)(mag >> 11)));  // ties to even; may reach 2^53
  if (E < -1021 || E > 1022) return ldexp(__ll2double_rn(S), q);     // near the ends of the range: slow path
  // the hidden bit of r adds one to the exponent field (two when r carried to 2^53)
  return __longlong_as_double((long long)(sign | (((uint64_t)(E + 1022) << 52) + r)));
}

// The same for q within +-1000, where no result leaves the normal range: about
// 25 integer instructions
__device__ __forceinline__ double fixed_to_double_inrange(long long S, int q) {
  const uint32_t neg = (uint32_t)((uint64_t)S >> 32) & 0x80000000u;
  const uint64_t mag = S < 0 ? 0ull - (uint64_t)S : (uint64_t)S;
  const uint32_t mh = (uint32_t)(mag >> 32), ml = (uint32_t)mag;
  const uint32_t h = mh ? mh : ml, l = mh ? ml : 0u;
  const int z = __clz((int)h);
  const uint32_t H = __funnelshift_l(l, h, z), L = l << z;   // leading one at bit 31 of H
  const uint32_t up = ((L & 0x7FFu) + ((L >> 11) & 1u) + 0x3FFu) >> 11;  // round to nearest even
  const uint32_t e = (uint32_t)((mh ? 1022 + 63 : 1022 + 31) - z + q);
  uint64_t r = ((uint64_t)(H >> 11) << 32) | __funnelshift_r(L, H, 11);
  r += ((uint64_t)(e << 20) << 32) + up;  // the hidden bit adds one to the exponent field
  r |= (uint64_t)neg << 32;
  return __longlong_as_double((long long)(h ? r : 0ull));
}

// d * 2^q for a finite double d, the exponent field adjusted as an integer
// when the result stays normal (else ldexp)
__device__ __forceinline__ double scale_pow2(double d, int q) {
  const uint64_t b = (uint64_t)__double_as_longlong(d);
  const int ex = (int)((b >> 52) & 0x7FF);
  if (ex == 0 || ex + q < 1 || ex + q > 2046) return ldexp(d, q);
  return __longlong_as_double((long long)(b + ((uint64_t)(int64_t)q << 52)));
}

}  // namespace
}  // namespace tn
