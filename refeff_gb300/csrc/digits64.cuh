// Signed 8-bit digits of FP64 values for exact products on the bf16 tensor
// path, and the conversion of their exact level sums back to FP64 (the scheme
// is described in tc_update64.cu; mma.sync form for small in-kernel updates
// below).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "cplx.cuh"

namespace rfx {

constexpr int kDig = 8;                 // digits per value
constexpr int kNonfinite = 1 << 28;     // exponent of a row or column with an infinity or NaN
constexpr int kNoEntry = -(1 << 20);    // exponent of a row or column of zeros

__device__ __forceinline__ int field_of(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
// larger exponent field of the two parts; -1 for zero (integer operations: a comparison on the FP64 pipe takes 16
// cycles a warp)
__device__ __forceinline__ int field_of(double2 v) {
  const int any = __double2loint(v.x) | __double2loint(v.y) | ((__double2hiint(v.x) | __double2hiint(v.y)) & 0x7fffffff);
  return any == 0 ? -1 : max(field_of(v.x), field_of(v.y));
}
// v 2^(62 - e) rounded to an integer (|v| < 2^e), biased by 128 in every byte: byte j holds digit 8 - j plus 128.
__device__ __forceinline__ uint2 biased_digits(double v, int e) {
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
  const int field = int(bits >> 52) & 0x7ff;
  unsigned long long x = bits & 0xfffffffffffffull;
  if (field) x |= 1ull << 52;
  const int sh = max(field, 1) - 1075 + 62 - e;  // <= 10
  if (sh >= 0) x <<= sh;
  else x = sh < -54 ? 0ull : (x + (1ull << (-sh - 1))) >> -sh;
  if (bits >> 63) x = 0ull - x;
  x += 0x8080808080808080ull;
  return make_uint2(uint32_t(x), uint32_t(x >> 32));
}
// digit d (0 .. 7, most significant first) as a float
__device__ __forceinline__ float digit_of(uint2 y, int d) {
  const int j = 7 - d;
  const uint32_t w = j >= 4 ? y.y : y.x;
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 | (j & 3))) - 8388736.0f;  // 2^23 + 128
}
// two small integers (exact in bf16: the high half of their FP32 patterns) as one bf16x2, a first
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// v 2^ex rounded to FP64 in integer operations, for results in the normal range (or zero): the conversion instruction
// runs on the FP64 pipe, where a warp's instruction takes 64 cycles of its quarter of the SM.
__device__ __forceinline__ double normal_double(long long v, int ex) {
  const uint32_t sign = uint32_t(static_cast<unsigned long long>(v) >> 32) & 0x80000000u;
  const unsigned long long a = static_cast<unsigned long long>(v < 0 ? -v : v);
  const int lz = __clzll(static_cast<long long>(a | 1));
  const unsigned long long m = a << lz;  // leading one at bit 63
  // 53 bits, rounded half up; a carry out of the mantissa moves into the exponent as it should
  const unsigned long long bits = (m >> 11) + ((m >> 10) & 1) + (static_cast<unsigned long long>(1023 + 62 - lz + ex) << 52);
  return v == 0 ? 0.0 : __hiloint2double(int(uint32_t(bits >> 32) | sign), int(uint32_t(bits)));
}
constexpr int kSafeExp = 900;  // sums of grids 2^e, |e| <= kSafeExp, are normal numbers
__device__ __forceinline__ double scaled_double(long long v, int ex) {
  return v == 0 || (ex >= -kSafeExp && ex <= kSafeExp) ? normal_double(v, ex) : scalbn(__ll2double_rn(v), ex);
}

// The grid's errors weigh some 2^-57 of 2^e in a sum of up to 32 complex products.  A sum below 2^(e - kWeak) beside a
// C below that may therefore have lost its terms; they are sound if the largest of them reaches 2^(e - kLost): the
// errors are then below 2^-49 of it, what the rounding of such a sum may come to.
constexpr int kWeak = 7, kLost = 6;
// both parts below 2^e (infinities and NaN are not)
__device__ __forceinline__ bool below(double2 v, int e) { return max(field_of(v.x), field_of(v.y)) < e + 1023; }

// The eight exact level sums of one real output (levels 2 .. 9, weights 2^-12 .. 2^-68 of 2^e, bit patterns of
// integer-valued floats) as an integer in units of 2^unit of 2^e: 2^-56, or 2^-68 where the sum lies below 2^-7 (the
// sum's grid is finer than FP64's there).  Integers up to 2^22 are read off the mantissa after adding 1.5 x 2^23, which
// holds for the levels 2 .. 6 at K = 32 (the first digit is at most 64).  kWide (K > 8): levels 7 and 8 can exceed that
// and are converted; level 9, up to 7/8 of 2^23, is read after adding 1.5 x 2^24, to an even integer.  The sum lies below
// 2^-kWeak where unit is kFineUnit.
constexpr int kFineUnit = -68;
template <bool kWide>
__device__ __forceinline__ long long join_levels(const uint32_t* s, int& unit) {
  constexpr uint32_t kBase = 0x4B400000u, kBase9 = 0x4BC00000u;  // the patterns of 1.5 x 2^23 and 1.5 x 2^24
  auto pat = [&](int i) { return __float_as_uint(__uint_as_float(s[i]) + 12582912.0f); };
  auto sum = [&](int i) { return kWide ? __float2int_rn(__uint_as_float(s[i])) : int(pat(i) - kBase); };
  const int p = int(pat(0) * 256u + pat(1) - 257u * kBase);
  const int q = int(pat(2) * 256u + pat(3) - 257u * kBase);
  const int r = int(pat(4) - kBase) * 256 + sum(5);
  const int l9 = kWide ? 2 * int(__float_as_uint(__uint_as_float(s[7]) + 25165824.0f) - kBase9) : int(pat(7) - kBase);
  const int l = sum(6) * 256 + l9;
  // h = the levels 2 .. 7 in units of 2^-56: |h| < 2^63; l holds levels 8 and 9, 12 bits further down
  const long long h = static_cast<long long>(p) * (1ll << 36) + static_cast<long long>(q) * (1 << 20) + static_cast<long long>(r) * 16;
  constexpr uint32_t kSmall = 1u << (56 - kWeak - 32);
  const bool small = uint32_t(static_cast<unsigned long long>(h) >> 32) + kSmall < 2 * kSmall;
  unit = small ? kFineUnit : -56;
  return small ? h * 4096 + l : h + ((l + 2048) >> 12);
}

// ---------------------------------------------------------------------------
// Warp-level form: C (16 x 8 complex) -= A (16 x 8) B (8 x 8) by mma.sync on the
// digits, for updates inside kernels that hold their operands in shared memory
// (too shallow, K = 8, to be worth a trip through tensor memory).  One
// m16n8k16 takes the real and imaginary parts of A side by side:
// Cr = [Ar Ai] [Br; -Bi], Ci = [Ar Ai] [Bi; Br].
// Lane (g = lane / 4, t = lane % 4) holds A[g or g + 8][2t, 2t + 1], B[2t, 2t + 1][g]
// and C[g or g + 8][2t, 2t + 1].
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct DigitTileA {
  uint32_t re[kDig][2], im[kDig][2];  // rows g and g + 8
  int e[2];                           // their exponents (kNoEntry: zeros)
};
// A column of A that lies 2^-s below the rows' largest entries in all 16 rows keeps 62 - s bits: a tile with one beyond
// this s (fewer than FP64's 53) is left to the FP64 pipe, as is one with an infinity or NaN.
constexpr int kTileSlack = 9;

// v[h][q] = A[g + 8 h][2t + q].  False (whole warp): the tile does not fit the digits.
__device__ __forceinline__ bool cut_tile_a(const double2 (&v)[2][2], DigitTileA& a) {
  int f[2][2], top[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    f[h][0] = field_of(v[h][0]);
    f[h][1] = field_of(v[h][1]);
    int t = max(f[h][0], f[h][1]);
    t = max(t, __shfl_xor_sync(0xffffffffu, t, 1));
    top[h] = max(t, __shfl_xor_sync(0xffffffffu, t, 2));
  }
  bool bad = top[0] == 0x7ff || top[1] == 0x7ff;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int m = max(f[0][q] > 0 ? f[0][q] - top[0] : -4096, f[1][q] > 0 ? f[1][q] - top[1] : -4096);
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 4));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
    bad = bad || (m < -kTileSlack && m > -4096);
  }
  if (__any_sync(0xffffffffu, bad)) return false;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    a.e[h] = top[h] < 0 ? kNoEntry : max(top[h], 1) - 1022;
    const int e = top[h] < 0 ? 0 : a.e[h];
    const uint2 r0 = biased_digits(v[h][0].x, e), r1 = biased_digits(v[h][1].x, e);
    const uint2 i0 = biased_digits(v[h][0].y, e), i1 = biased_digits(v[h][1].y, e);
#pragma unroll
    for (int d = 0; d < kDig; ++d) {
      a.re[d][h] = pack_bf16(digit_of(r0, d), digit_of(r1, d));
      a.im[d][h] = pack_bf16(digit_of(i0, d), digit_of(i1, d));
    }
  }
  return true;
}

// Digits of B for one 8-column group, stored as words [2 d + part][lane] (part 0 re, 1 im) and the column exponents;
// v[q] = B[2t + q][g].  A column with an infinity or NaN gets the exponent kNonfinite, one of zeros kNoEntry.
__device__ __forceinline__ void cut_tile_b(const double2 (&v)[2], uint32_t* words, int* ecol) {
  const int lane = threadIdx.x & 31;
  int t = max(field_of(v[0]), field_of(v[1]));
  t = max(t, __shfl_xor_sync(0xffffffffu, t, 1));
  t = max(t, __shfl_xor_sync(0xffffffffu, t, 2));
  if ((lane & 3) == 0) ecol[lane >> 2] = t == 0x7ff ? kNonfinite : t < 0 ? kNoEntry : max(t, 1) - 1022;
  const bool bad = t == 0x7ff || t < 0;
  const int e = bad ? 0 : max(t, 1) - 1022;
  const uint2 r0 = biased_digits(bad ? 0.0 : v[0].x, e), r1 = biased_digits(bad ? 0.0 : v[1].x, e);
  const uint2 i0 = biased_digits(bad ? 0.0 : v[0].y, e), i1 = biased_digits(bad ? 0.0 : v[1].y, e);
#pragma unroll
  for (int d = 0; d < kDig; ++d) {
    words[(2 * d) * 32 + lane] = pack_bf16(digit_of(r0, d), digit_of(r1, d));
    words[(2 * d + 1) * 32 + lane] = pack_bf16(digit_of(i0, d), digit_of(i1, d));
  }
}

// p[h][q] = sum_k A[g + 8 h][k] B[k][2t + q] of the digits in `a` and of the words of cut_tile_b, on the grid
// 2^(a.e[h] + ecol[2t + q]).  Bit 2 h + q of the result: the sum lies below 2^-kWeak of it.
__device__ __forceinline__ uint32_t tile_product(const DigitTileA& a, const uint32_t* words, const int* ecol,
                                                 double2 (&p)[2][2]) {
  const int lane = threadIdx.x & 31, t = lane & 3;
  float cr[kDig][4], ci[kDig][4];
#pragma unroll
  for (int s = 0; s < kDig; ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i) cr[s][i] = ci[s][i] = 0.f;
#pragma unroll
  for (int j = 0; j < kDig; ++j) {
    const uint32_t br = words[(2 * j) * 32 + lane], bi = words[(2 * j + 1) * 32 + lane], nbi = bi ^ 0x80008000u;
#pragma unroll
    for (int i = 0; i + j < kDig; ++i) {
      mma_k16(cr[i + j], a.re[i][0], a.re[i][1], a.im[i][0], a.im[i][1], br, nbi);
      mma_k16(ci[i + j], a.re[i][0], a.re[i][1], a.im[i][0], a.im[i][1], bi, br);
    }
  }
  uint32_t weak = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t lr[kDig], li[kDig];
#pragma unroll
      for (int s = 0; s < kDig; ++s) {
        lr[s] = __float_as_uint(cr[s][2 * h + q]);
        li[s] = __float_as_uint(ci[s][2 * h + q]);
      }
      const int e = a.e[h] + ecol[2 * t + q];
      int ur, ui;
      const long long vr = join_levels<false>(lr, ur);
      p[h][q].x = scaled_double(vr, e + ur);
      const long long vi = join_levels<false>(li, ui);
      p[h][q].y = scaled_double(vi, e + ui);
      if (ur + ui == 2 * kFineUnit && e > kNoEntry / 2) weak |= 1u << (2 * h + q);  // else a row or column of zeros
    }
  return weak;
}

}  // namespace rfx
