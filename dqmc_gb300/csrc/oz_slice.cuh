// Exact slicing of FP64 values into BF16 digits for the split-precision GEMM
// (k_ozaki.cu).  The delayed local-update kernel (k_local.cu) uses the same
// code to slice its own rows of the pending factors at the end of a round.
#pragma once
#include <cuda_bf16.h>
#include "common.cuh"
#include "kernels.h"

// The slicing runs on the integer units.  A row (column) scale is 2^E with
// E the frexp exponent of its largest |Re|/|Im|, taken from the exponent
// fields; x 2^-E (|.| < 1) becomes a 62-bit fixed-point integer built from
// the mantissa, and the S signed digits are cut off it by shifts.
__device__ __forceinline__ int expo_field(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7FF);
}

// x 2^(62 - E) as an integer (|x| < 2^E); values below 2^(E-62) are dropped
__device__ __forceinline__ long long fixed62(double x, int E) {
  const long long b = __double_as_longlong(x);
  const int ef = (int)((b >> 52) & 0x7FF);
  if (ef == 0) return 0;
  const long long m = (b & 0xFFFFFFFFFFFFFll) | 0x10000000000000ll;   // x = m 2^(ef - 1075)
  const int sh = ef - 1075 - E + 62;                                   // <= 9
  long long X = 0;
  if (sh >= 0) X = m << sh;
  else if (sh > -63) X = m >> (-sh);
  return b < 0 ? -X : X;
}

// Cuts the next signed digit off a 62-bit fixed-point integer: X / 2^s rounded
// half to even, X <- X - digit 2^s (so |digit| <= 2^bits for the first and
// 2^(bits - 1) for the later ones).  s < 0 only for the last of 8 slices of 8 bits
// and of 9 of 7.
__device__ __forceinline__ int oz_next_digit(long long& X, int s) {
  if (s <= 0) {
    const long long d = X * (1ll << -s);
    X = 0;
    return (int)d;
  }
  // + half a unit, less one unit of X's last place when the floor is even
  const long long q = (X + ((1ll << (s - 1)) - 1) + ((X >> s) & 1)) >> s;
  X -= q << s;
  return (int)q;
}

// The scale of a vector whose largest exponent field is me: 2^E > max |.| with E
// the frexp exponent, stored as 2^(E-1) (finite for every finite vector); NaN
// when the vector holds an Inf or a NaN, so that every output it enters is NaN.
__device__ __forceinline__ int oz_scale_expo(int me) { return me > 0 ? me - 1022 : 0; }
__device__ __forceinline__ double oz_scale_value(int me) {
  if (me == 0x7FF) return __longlong_as_double(0x7FF8000000000000ll);
  return __longlong_as_double((long long)(oz_scale_expo(me) - 1 + 1023) << 52);
}

__device__ __forceinline__ uint32_t oz_pack2(int a, int b) {   // two digits as BF16 (exact), a at the lower address
  const __nv_bfloat162 v = __floats2bfloat162_rn((float)a, (float)b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// |x| 2^-E (< 1) as BF16, truncated; 0 only for x = 0 (below 2^-60: 2^-60).
__device__ __forceinline__ uint32_t oz_mag(double x, int E) {
  const long long b = __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll;
  if (b == 0) return 0u;
  const int f = (int)(b >> 52) - 1023 - E + 127;
  return f < 67 ? 67u << 7 : (uint32_t)f << 7 | ((uint32_t)(b >> 45) & 0x7Fu);
}

// Digits of the entries k, k + 1 (k even) of vector vec of one side of a
// product into o: side 0 a row of op(A) (As: Re digits in k, Im digits in
// Kpad + k), side 1 a column of op(B) (B'_re = [Re; -Im], B'_im = [Im; Re]).
// With Bmag the magnitudes as well (side 0 |Re|, |Im| as slice S of As; side 1
// the larger of the two in both halves).
__device__ __forceinline__ void oz_store_pair(const OzSlices& o, int side, int vec, int k, cplx x0, cplx x1, int E) {
  const size_t Kp = 2 * (size_t)o.Kpad;
  long long r0 = fixed62(x0.x, E), i0 = fixed62(x0.y, E), r1 = fixed62(x1.x, E), i1 = fixed62(x1.y, E);
  for (int p = 0; p < o.S; ++p) {
    const int s = 62 - (p + 1) * o.bits;
    const int a0 = oz_next_digit(r0, s), a1 = oz_next_digit(r1, s);
    const int b0 = oz_next_digit(i0, s), b1 = oz_next_digit(i1, s);
    if (side == 0) {
      __nv_bfloat16* a = o.As + (size_t)p * o.m * Kp + (size_t)vec * Kp;
      *reinterpret_cast<uint32_t*>(a + k) = oz_pack2(a0, a1);
      *reinterpret_cast<uint32_t*>(a + o.Kpad + k) = oz_pack2(b0, b1);
    } else {
      const size_t base = (size_t)p * o.n * Kp + (size_t)vec * Kp;
      const uint32_t re = oz_pack2(a0, a1), im = oz_pack2(b0, b1);
      *reinterpret_cast<uint32_t*>(o.Bre + base + k) = re;
      *reinterpret_cast<uint32_t*>(o.Bre + base + o.Kpad + k) = oz_pack2(-b0, -b1);
      *reinterpret_cast<uint32_t*>(o.Bim + base + k) = im;
      *reinterpret_cast<uint32_t*>(o.Bim + base + o.Kpad + k) = re;
    }
  }
  if (o.Bmag) {
    const uint32_t re = oz_mag(x0.x, E) | oz_mag(x1.x, E) << 16, im = oz_mag(x0.y, E) | oz_mag(x1.y, E) << 16;
    __nv_bfloat16* v = side == 0 ? o.As + (size_t)o.S * o.m * Kp + (size_t)vec * Kp : o.Bmag + (size_t)vec * Kp;
    const uint32_t mx = __vmaxu2(re, im);   // BF16 of non-negative values order like integers
    *reinterpret_cast<uint32_t*>(v + k) = side == 0 ? re : mx;
    *reinterpret_cast<uint32_t*>(v + o.Kpad + k) = side == 0 ? im : mx;
  }
}

// One warp slices vector vec: x(k) gives its entries for k < K; zeros are
// written up to Kpad, and the scale goes to sA / sB.
template <class Get>
__device__ __forceinline__ void oz_slice_vec(const OzSlices& o, int side, int vec, int K, Get x, int lane) {
  int me = 0;
  for (int k = lane; k < K; k += 32) {
    const cplx v = x(k);
    me = max(me, max(expo_field(v.x), expo_field(v.y)));
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) me = max(me, __shfl_xor_sync(0xffffffffu, me, s));
  if (lane == 0) (side ? o.sB : o.sA)[vec] = oz_scale_value(me);
  const int E = oz_scale_expo(me);
  for (int k = 2 * lane; k < o.Kpad; k += 64) {
    const cplx x0 = k < K ? x(k) : cmake(0.0, 0.0), x1 = k + 1 < K ? x(k + 1) : cmake(0.0, 0.0);
    oz_store_pair(o, side, vec, k, x0, x1, E);
  }
}
