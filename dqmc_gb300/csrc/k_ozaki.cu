// Split-precision complex GEMM on the BF16 tensor cores (Ozaki scheme).
//
//   C = alpha * diag(rs) * op(A) * op(B) * diag(cs) + beta * C     (complex FP64)
//
// GB300 runs FP64 at ~1/1500 of its BF16 tensor rate, so both forms compute the
// dense products of the UDT stabilisation and of the local updates' flush as
// sums of exact BF16 x BF16 -> FP32 products:
//
//  * every row i of op(A) gets a power-of-two scale sigma_i > max_k |op(A)_ik|
//    (real and imaginary parts together), every column j of op(B) a scale
//    tau_j; the scaled entries lie in (-1, 1);
//  * each scaled entry x is cut into S slices of B bits, x ~ sum_p 2^{-B p} a_p
//    with integers |a_1| <= 2^B, |a_p| <= 2^(B-1), which BF16 holds exactly;
//  * the complex product is two real GEMMs with K' = 2K on stacked operands,
//    A' = [Re A, Im A] and B'_re = [Re B; -Im B], B'_im = [Im B; Re B];
//  * slice pairs (p, q) with p + q = t <= S + 1 are accumulated into one FP32
//    accumulator per t, over chunks of K' short enough that
//    chunk (S + 2) 2^{2B - 2} <= 2^24 (the digit bounds above, summed over the
//    pairs of a group): every partial sum is an integer of at most 24 bits, so
//    the FP32 accumulation is exact whatever K is (S = 9 slices of 7 bits, the
//    FP64 form's products: chunks of 320);
//  * the group sums of all chunks are combined exactly in 64-bit integers (one
//    for up to 61 bits, else a high and a low one) and the result is rounded once
//    to double with its power-of-two weight and the scales.
// The errors besides that rounding are the truncation of the slice expansion
// (2^{-B S - 1}, at least 2^{-62}, relative to sigma_i and tau_j) and the dropped
// pairs p + q > S + 1 of the same size.  They go by the largest entries of row i
// and column j: an entry far below them has fewer bits than in FP64.
//
// FP64 form (S = 9, "full"): below 2^-65 sqrt(2 K) sigma_i tau_j, where an FMA
// chain's error is about 2^-54.5 M, M = sum_k |a_ik| |b_kj|.  That is 0.003 of it for
// random entries (M = sqrt(2 K) / 4 in units of the scales; K = 16 .. 1024, exact
// integers) and more than all of it below M = sqrt(2 K) / 2000, where the large
// entries of the row meet the small ones of the column.  Products whose elements
// are to be as good as FMA chains one by one (operands from the caller, the LU's
// and the triangular solves' updates) are guarded: one BF16 magnitude per entry (a
// float with its own exponent, down to 2^-60) is kept beside the slices, the tensor
// cores sum M from them to 1%, and where M < 2^-8 sqrt(2 K) sigma_i tau_j (and the
// sum with an old C is below that, too) the element is an FP64 dot product of the
// operands instead (oz_dot).  At that limit the slices' error is 0.2 of the FMA
// chain's.  The magnitudes are one more A tile per K block, a twelfth more of B and
// 1 / 45 of the arithmetic.  Rows and columns with an Inf or NaN are dot products in
// every full product, as long as it has its operands.
// The tensor-core products run on tcgen05.mma (kind::f16, BF16 in, FP32
// accumulators in tensor memory), with every operand tile staged by TMA
// (cp.async.bulk.tensor) onto mbarriers; see the engine section below.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <algorithm>
#include "common.cuh"
#include "kernels.h"
#include "oz_slice.cuh"

namespace {

// ---------------------------------------------------------------------------
// split: slices of op(X) scaled per row ("row" side = A) or per column (B side)
// ---------------------------------------------------------------------------
// (the digit helpers are in oz_slice.cuh)

// Slices of both operands in one launch: blockIdx.y = 0 rows of op(A), 1
// columns of op(B), SPLIT_V vectors per CTA, two warps per vector.  The
// vectors are read from global memory once, into shared memory, along the
// direction in which X is contiguous (op(A) = A and op(B) = B^T, B^C: across
// the vectors; otherwise along a vector); the scales and the digits are then
// cut from shared memory, two entries per lane so that every store of a warp
// is 128 contiguous bytes.  At 1024 x 1024 the two one-vector-per-CTA kernels
// this replaces read X twice, with one 16-byte word per 16 KB stride on the
// strided side.
constexpr int SPLIT_V = 4;
__global__ void __launch_bounds__(64 * SPLIT_V) k_oz_split(const cplx* __restrict__ A, int lda, char opA,
                                                           const cplx* __restrict__ B, int ldb, char opB, int K,
                                                           OzSlices o) {
  extern __shared__ double4_16a smem_split[];
  cplx* tile = reinterpret_cast<cplx*>(smem_split);   // (SPLIT_V, K + 1)
  __shared__ int s_me[2 * SPLIT_V];
  const int side = blockIdx.y;
  const cplx* X = side ? B : A;
  const int ld = side ? ldb : lda, cnt = side ? o.n : o.m;
  const char op = side ? opB : opA;
  const int v0 = blockIdx.x * SPLIT_V;
  if (v0 >= cnt) return;
  const int ldt = K + 1;
  const bool across = side ? op != 'N' : op == 'N';   // X contiguous across the vectors
  const bool conj = op == 'C';
  if (across) {
    for (int e = threadIdx.x; e < K * SPLIT_V; e += blockDim.x) {
      const int k = e / SPLIT_V, v = e % SPLIT_V;
      cplx x = v0 + v < cnt ? X[(size_t)k * ld + v0 + v] : cmake(0.0, 0.0);
      tile[v * ldt + k] = conj ? cconj(x) : x;
    }
  } else {
    for (int v = 0; v < SPLIT_V && v0 + v < cnt; ++v)
      for (int k = threadIdx.x; k < K; k += blockDim.x) {
        const cplx x = X[(size_t)(v0 + v) * ld + k];
        tile[v * ldt + k] = conj ? cconj(x) : x;
      }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int v = wid >> 1, half = wid & 1;
  const bool live = v0 + v < cnt;
  const cplx* x = tile + v * ldt;
  int me = 0;
  if (live)
    for (int k = 32 * half + lane; k < K; k += 64) me = max(me, max(expo_field(x[k].x), expo_field(x[k].y)));
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) me = max(me, __shfl_xor_sync(0xffffffffu, me, s));
  if (lane == 0) s_me[wid] = me;
  __syncthreads();
  if (!live) return;
  me = max(s_me[2 * v], s_me[2 * v + 1]);
  if (half == 0 && lane == 0) (side ? o.sB : o.sA)[v0 + v] = oz_scale_value(me);
  const int E = oz_scale_expo(me);
  for (int k = 64 * half + 2 * lane; k < o.Kpad; k += 128)
    oz_store_pair(o, side, v0 + v, k, k < K ? x[k] : cmake(0.0, 0.0), k + 1 < K ? x[k + 1] : cmake(0.0, 0.0), E);
}

struct OzArgs {
  const cplx *A, *B;         // full form: the operands, op(A) (m x k) and op(B) (k x n) (null: sliced elsewhere)
  int lda, ldb, k;
  char opA, opB;
  float theta;               // guarded: the least magnitude sum (in units of the scales) that the slices carry
  int theta_e;               // ceil(log2(theta))
  const double* sA;          // (m) row scales 2^(E-1)
  const double* sB;          // (n) column scales
  int m, n, Kp, S, bits;
  cplx alpha, beta;
  cplx* C;
  int ldc;
  const double* rs;          // optional extra row scaling
  const double* cs;          // optional extra column scaling
  const int* active;         // optional: nothing to do when *active == 0
  int kexact;                // K blocks per exact accumulation (chunk)
  int kchunk;                // split K: K blocks per CTA layer (blockIdx.z); 0 = all
  unsigned long long* acc;   // split K: exact integer sums (m x n x {re, im}, wide: {re hi, re lo, im hi, im lo},
                             // guarded: and the magnitudes in 2^-40, rounded up),
                             // finished by k_oz_finalize (zero on entry; the finaliser zeroes what it read)
};

// alpha v + beta c_old for one output value (the scaled product v):
// alpha = +-1, beta in {0, 1} take one multiply and at most one add.
__device__ __forceinline__ cplx oz_combine(const OzArgs& a, cplx beta, cplx v, cplx c_old, bool plain) {
  if (plain) {
    if (a.alpha.x < 0.0) v = cmake(-v.x, -v.y);
    if (beta.x != 0.0) v = cadd(c_old, v);
    return v;
  }
  v = cmul(a.alpha, v);
  if (beta.x != 0.0 || beta.y != 0.0) v = cfma(beta, c_old, v);
  return v;
}

__device__ __forceinline__ bool oz_plain(const OzArgs& a) {
  return (a.alpha.x == 1.0 || a.alpha.x == -1.0) && a.alpha.y == 0.0 && a.beta.y == 0.0 &&
         (a.beta.x == 0.0 || a.beta.x == 1.0);
}

// The exact value of a wide sum is hi 2^WIDE_SHIFT(bits) + lo.
__host__ __device__ constexpr int oz_wide_groups() { return 4; }   // groups of the low word
__device__ __forceinline__ int oz_wide_shift(int bits) { return oz_wide_groups() * bits; }

// (double)v 2^e, rounded to nearest even exactly as __ll2double_rn(v) * 2^e,
// on the integer units and without branches, for -1022 <= e <= 960 (every
// |v| < 2^63 then gives a normal double): |v| is shifted so that its leading
// one sits at bit 63, the 53 high bits are rounded to nearest even at bit 11,
// and a carry out of the significand steps the biased exponent by addition.
__device__ __forceinline__ double ll_ldexp(long long v, int e) {
  const unsigned long long sgn = (unsigned long long)v & 0x8000000000000000ull;
  const unsigned long long m = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)m) & 63;   // 64 for m = 0, masked; the select below covers it
  const unsigned long long mn = m << lz;
  unsigned long long q = mn >> 11;
  const unsigned rem = (unsigned)mn & 0x7FFu;
  q += (rem + (unsigned)(q & 1ull)) > 0x400u ? 1ull : 0ull;
  const long long be = 63 - lz + e + 1023;
  const unsigned long long bits = sgn | ((unsigned long long)(be - 1) << 52) + q;
  return m ? __longlong_as_double((long long)bits) : 0.0;
}

// The same for the exact sum hi 2^sh + lo (|sum| < 2^100, sh < 64), rounded
// once: the 128-bit magnitude is normalised to bit 127 and the words below
// the rounding position enter as a sticky bit.  Normal results for
// -1022 <= e <= 900.
__device__ __forceinline__ double wide_ldexp(long long hi, long long lo, int sh, int e) {
  const unsigned long long h0 = (unsigned long long)hi;
  unsigned long long l = h0 << sh;
  unsigned long long h = (unsigned long long)(hi >> (64 - sh));
  l += (unsigned long long)lo;
  h += (unsigned long long)(lo >> 63) + (l < (unsigned long long)lo ? 1ull : 0ull);
  const bool neg = (long long)h < 0;
  if (neg) {
    l = 0ull - l;
    h = ~h + (l == 0ull ? 1ull : 0ull);
  }
  int ex = e + 64;
  if (h == 0ull) { h = l; l = 0ull; ex = e; }
  const int lz = __clzll((long long)h) & 63;
  const unsigned long long m = lz ? (h << lz) | (l >> (64 - lz)) : h;
  const bool sticky = (l << lz) != 0ull;
  unsigned long long q = m >> 11;
  const unsigned rem = (unsigned)m & 0x7FFu;
  q += (rem + ((unsigned)(q & 1ull) | (sticky ? 1u : 0u))) > 0x400u ? 1ull : 0ull;
  const long long be = 63 - lz + ex + 1023;
  const unsigned long long bits = (neg ? 0x8000000000000000ull : 0ull) | ((unsigned long long)(be - 1) << 52) + q;
  return h ? __longlong_as_double((long long)bits) : 0.0;
}

// An exact sum times 2^e.  window: e lies where every sum gives a normal
// double (integer route); otherwise the FP64 route with its range handling.
template <bool WIDE>
__device__ __forceinline__ double oz_value(long long hi, long long lo, int sh, int e, bool window) {
  if constexpr (WIDE) {
    if (window) return wide_ldexp(hi, lo, sh, e);
    return ldexp(wide_ldexp(hi, lo, sh, 0), e);
  } else {
    if (window) return ll_ldexp(hi, e);
    return ldexp(__ll2double_rn(hi), e);
  }
}
__device__ __forceinline__ bool oz_window(int e) { return e >= -1022 && e <= 900; }
constexpr int OZ_EXPO_NAN = 1 << 20;   // exponent of a NaN scale: no window, NaN results
__device__ __forceinline__ int oz_expo(double scale) {   // E of the stored scale 2^(E-1)
  const int f = expo_field(scale);
  return f == 0x7FF ? OZ_EXPO_NAN : f - 1022;
}

// ---- full form: elements that the slices do not carry ----
// Whether the slices carry an element of value v (old C included) and magnitude
// sum mag, scales 2^ex: mag or, where v is a sum with the old C (sum), v itself is
// large enough.  mag = 0: no term differs from zero.  Not finite: as k_zgemm has it.
template <bool GUARD>
__device__ __forceinline__ bool oz_carried(const OzArgs& a, float mag, int ex, cplx v, bool sum) {
  const int f = max(expo_field(v.x), expo_field(v.y));
  if (f == 0x7FF || ex > OZ_EXPO_NAN / 2) return false;
  return !GUARD || mag >= a.theta || mag == 0.0f || (sum && f > 1023 + ex + a.theta_e);
}
// extra scalings one after the other (their product could leave the range of double)
__device__ __forceinline__ cplx oz_scale2(const OzArgs& a, cplx v, int row, int col) {
  if (a.rs) v = cscale(v, a.rs[row]);
  if (a.cs) v = cscale(v, a.cs[col]);
  return v;
}
// t = op(A)[row, :] op(B)[:, col] into C[row, col], as k_zgemm does (also for what is not finite)
__device__ __forceinline__ void oz_put(const OzArgs& a, int row, int col, cplx t) {
  cplx* cp = &a.C[(size_t)col * a.ldc + row];
  t = cmul(a.alpha, oz_scale2(a, t, row, col));
  if (a.beta.x != 0.0 || a.beta.y != 0.0) t = cfma(a.beta, *cp, t);
  *cp = t;
}
// The elements C[row of this lane, col] for which need is set: dot products in
// FP64 multiply-adds over the operands (called by whole warps; C still holds its
// old value there).  8 lanes per element, or one where most lanes have one; every
// lane adds four sums and reads four terms ahead.  Bound: FP64 issue, 4 multiply-
// adds per term as for k_zgemm, and with 8 lanes as much again for the sums of the
// lanes at K = 64.  All elements of n = 1024: not read ahead 17.1 ms, so 10.1
// (k_zgemm 8.3).
__device__ __forceinline__ void oz_dot(const OzArgs& a, int row, int col, bool need) {
  const int lane = threadIdx.x & 31, K = a.k;
  const size_t sa = a.opA == 'N' ? a.lda : 1, sb = a.opB == 'N' ? 1 : a.ldb;
  const int fa = a.opA == 'C' ? (int)0x80000000 : 0, fb = a.opB == 'C' ? (int)0x80000000 : 0;
  auto conj_if = [](cplx v, int f) { return cmake(v.x, __hiloint2double(__double2hiint(v.y) ^ f, __double2loint(v.y))); };
  unsigned todo = __ballot_sync(0xffffffffu, need);
  const bool lanes = __popc(todo) >= 20;   // one lane per element
  while (todo) {
    int r = row, c = col, k0 = 0, step = 1;
    bool on = need;
    if (lanes) {
      todo = 0u;
    } else {
      int src = -1;   // lane group q takes the q-th element left
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (todo && lane >> 3 == q) src = __ffs(todo) - 1;
        todo &= todo - 1;
      }
      on = src >= 0;
      r = __shfl_sync(0xffffffffu, row, max(src, 0));
      c = __shfl_sync(0xffffffffu, col, max(src, 0));
      k0 = lane & 7;
      step = 8;
    }
    cplx s[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = cmake(0.0, 0.0);
    if (on) {
      const cplx* pa = a.opA == 'N' ? a.A + r : a.A + (size_t)r * a.lda;
      const cplx* pb = a.opB == 'N' ? a.B + (size_t)c * a.ldb : a.B + c;
      cplx x[4], y[4], xn[4], yn[4];
      auto read = [&](int k, cplx(&u)[4], cplx(&v)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int kk = k + q * step;
          u[q] = kk < K ? pa[kk * sa] : cmake(0.0, 0.0);
          v[q] = kk < K ? pb[kk * sb] : cmake(0.0, 0.0);
        }
      };
      read(k0, x, y);
#pragma unroll 1
      for (int k = k0; k < K; k += 4 * step) {
        read(k + 4 * step, xn, yn);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          s[q] = cfma(conj_if(x[q], fa), conj_if(y[q], fb), s[q]);
          x[q] = xn[q];
          y[q] = yn[q];
        }
      }
    }
    cplx t = cadd(cadd(s[0], s[1]), cadd(s[2], s[3]));
    if (!lanes) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
        t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
      }
    }
    if (on && (lanes || (lane & 7) == 0)) oz_put(a, r, c, t);
    __syncwarp();
  }
}

template <bool WIDE, bool FULL = false, bool GUARD = false>
__global__ void k_oz_finalize(OzArgs a) {
  const int e0 = -a.bits * (a.S + 1), sh = oz_wide_shift(a.bits);
  const bool plain = oz_plain(a);
  const size_t total = (size_t)a.m * a.n;
  constexpr int W = WIDE ? 2 : 1, WORDS = 2 * W + (GUARD ? 1 : 0);
  // whole warps stay in the loop (oz_dot)
  for (size_t b = (size_t)blockIdx.x * blockDim.x; b < total; b += (size_t)gridDim.x * blockDim.x) {
    const size_t e = b + threadIdx.x;
    const bool in = e < total;
    const int col = in ? (int)(e / a.m) : 0, row = in ? (int)(e - (size_t)col * a.m) : 0;
    bool need = false;
    if (in) {
      long long v[WORDS];
#pragma unroll
      for (int q = 0; q < WORDS; ++q) {
        v[q] = (long long)a.acc[WORDS * e + q];
        a.acc[WORDS * e + q] = 0ull;
      }
      const int ex = oz_expo(a.sA[row]) + oz_expo(a.sB[col]);
      cplx r = cmake(oz_value<WIDE>(v[0], v[W - 1], sh, e0 + ex, oz_window(e0 + ex)),
                     oz_value<WIDE>(v[W], v[2 * W - 1], sh, e0 + ex, oz_window(e0 + ex)));
      if (ex > OZ_EXPO_NAN / 2) r = cmake(nan(""), nan(""));
      if constexpr (FULL) r = oz_scale2(a, r, row, col);
      else if (a.rs || a.cs) r = cscale(r, (a.rs ? a.rs[row] : 1.0) * (a.cs ? a.cs[col] : 1.0));
      cplx* cp = &a.C[(size_t)col * a.ldc + row];
      const bool rd = a.beta.x != 0.0 || a.beta.y != 0.0;
      r = oz_combine(a, a.beta, r, rd ? *cp : cmake(0.0, 0.0), plain);
      if constexpr (FULL)
        need = a.A && !oz_carried<GUARD>(a, GUARD ? (float)v[WORDS - 1] * 0x1p-40f : 0.0f, ex, r,
                                         rd && plain && !a.rs && !a.cs);
      if (!need) *cp = r;
    }
    if constexpr (FULL) oz_dot(a, row, col, need);
  }
}

// ---------------------------------------------------------------------------
// tcgen05 engine: TMA-staged slices, tensor-core MMAs into TMEM accumulators
// ---------------------------------------------------------------------------
// A CTA computes 128 x BN complex tiles of C (BN = 32, 16 or 8, in the full form
// 24, 16 or 8; the figures below are for 32), persistently: one CTA per SM
// takes tiles x, x + grid, ... and the MMAs of a tile run while the epilogue
// of the previous one converts and stores.  Each MMA is
// M = 128, K = 16 (kind::f16, BF16 in, FP32 out), N = 64 per B slice: the
// slice's tile stacks the 32 columns of B'_re over the 32 of B'_im, so one
// accumulator holds [Re | Im] of the tile.  Every group t = p + q (2 <= t <= S + 1) has
// its own accumulator of 64 TMEM columns, all S live at once (S <= 8: 512
// columns), so one pass over K serves every slice pair and each K block of
// every slice is staged once:
//   * warp 0 (one lane) streams, per K block of 64 of every tile, the S
//     B-slices (double-buffered) and the S A-slices (a ring of 6) with
//     cp.async.bulk.tensor (128-byte swizzle) onto mbarriers;
//   * warp 1 allocates TMEM, and one lane issues tcgen05.mma for every pair
//     (p, q) with p + q <= S + 1 into group p + q, releasing each A slot and
//     B buffer with tcgen05.commit and marking a chunk's accumulators final
//     with a commit; before the first MMA of the next chunk (of this tile or
//     the next) it waits until the epilogue has read them out of TMEM;
//   * the other warps (four per TMEM lane quarter, 8 columns each) read the S
//     exact FP32 group sums of a chunk with tcgen05.ld, release TMEM, add
//     the sums with their weights to 64-bit integers (two words above 61 bits),
//     and after the tile's last chunk round, scale and store.
// The full form (S = 9) has tiles of at most 24 columns, so that its 9 groups of
// 48 columns (and the magnitudes' 32, if guarded) fit into TMEM; the magnitudes are
// slice S of A and one more B tile, summed over all chunks of a tile.  At n = 1024,
// slicing included, 8 slices of 7 bits at 32 columns -> this: product 0.36 -> 0.48 ms,
// flush of 16 sites 36 -> 44 us on average.
// Every wait is bounded; on a timeout the kernel sets an error bit, drains
// what it issued (bounded) and frees its TMEM.
constexpr int TC_BM = 128;                      // rows of C per CTA (TMEM lanes)
constexpr int TC_BN = 32;                       // complex columns of C per tile, at most (BN of the kernel: 32, 16 or 8)
constexpr int TC_BK = 64;                       // BF16 per K block: one 128-byte swizzle row
constexpr int TC_MAXS = 8;                      // S groups x 64 TMEM columns <= 512
constexpr int TC_BN_FULL = 24;                 // widest tile of the full form: 9 x 48 + 32 TMEM columns
// columns of the magnitude product (N of an MMA with M = 128 is a multiple of 16)
__host__ __device__ constexpr int tc_mag_cols(int bn) { return (bn + 15) / 16 * 16; }
constexpr int TC_ARING = 6;                     // A-slice stages (S <= 6: one K block of A in flight)
// epilogue warps, from 2 on: four per TMEM lane quarter, BN / 4 columns each; three of 8
// columns at BN = 24 (with 16 warps of 6 a thread has 96 registers and spills)
__host__ __device__ constexpr int tc_epi_warps(int bn) { return bn == 24 ? 12 : 16; }
__host__ __device__ constexpr int tc_threads(int bn) { return 32 * (2 + tc_epi_warps(bn)); }   // warp 0 TMA, warp 1 MMA
constexpr int TC_A_TILE = TC_BM * TC_BK * 2;    // 16 KB
__host__ __device__ constexpr int tc_b_half(int bn) { return bn * TC_BK * 2; }   // 4 KB at BN = 32: BN rows of B'_re or of B'_im
// MMA instruction descriptor (kind::f16): D F32 (bits 4-5 = 1), A BF16 (bits
// 7-9 = 1), B BF16 (bits 10-12 = 1), both K-major (bits 15, 16 = 0),
// N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)n >> 3 << 17) | ((uint32_t)TC_BM >> 4 << 24);
}
// B slices of one MMA.  For a fixed A slice p the pairs (p, q), q = 0, 1, ...
// write adjacent groups of 64 TMEM columns, and the B slices' tiles of 64 rows
// are adjacent in shared memory, so up to 4 of them (at BN = 32) are one MMA of N = 256: the
// tensor core then reads A (4 KB per K step) once for them.  At N = 64 the 6 KB
// of operands per MMA took 48 cycles of shared-memory bandwidth for 32 of
// arithmetic.
__host__ __device__ constexpr int tc_nstack(int bn) { return 128 / bn; }

// B slices of one K block (and the magnitudes, mag columns of them)
__host__ __device__ constexpr int tc_b_bytes(int S, int bn, int mag) { return 2 * S * tc_b_half(bn) + mag * TC_BK * 2; }
__host__ __device__ constexpr size_t tc_smem_bytes(int S, int bn, int mag) {
  return 1024 + (size_t)2 * tc_b_bytes(S, bn, mag) + (size_t)TC_ARING * TC_A_TILE + 256;
}
static_assert(tc_smem_bytes(9, TC_BN_FULL, tc_mag_cols(TC_BN_FULL)) <= 227 * 1024, "shared memory of a CTA");
__host__ __device__ constexpr uint32_t tc_tmem_cols(int cols) {   // a power of two
  return cols <= 32 ? 32u : (cols <= 64 ? 64u : (cols <= 128 ? 128u : (cols <= 256 ? 256u : 512u)));
}

// Shared-memory matrix descriptor of a K-major operand tile written by TMA
// with the 128-byte swizzle: start address >> 4 (bits 0-13), leading byte
// offset 16 >> 4 (bits 16-29; unused for this layout), stride byte offset
// 1024 >> 4 between 8-row groups (bits 32-45), descriptor version 1 (bits
// 46-47), layout SWIZZLE_128B = 2 (bits 61-63).  Tiles start on 1024-byte
// boundaries; the K step of 16 BF16 (32 bytes) inside the swizzle row adds
// 2 to the start field.
__device__ __forceinline__ uint64_t tc_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// Waits until the phase of parity `parity` of the barrier has completed; gives
// up after ~2^31 SM cycles (about a second), sets the error bit and *abort.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* err, volatile int* abort) {
  const long long t0 = clock64();
  for (uint32_t it = 0;; ++it) {
    if (mbar_test(bar, parity)) return true;
    if ((it & 255) == 255) {
      if (*abort) return false;
      if (clock64() - t0 > (1ll << 31)) {
        atomicOr(err, DQMC_KERR_BARRIER_TIMEOUT);
        *abort = 1;
        return false;
      }
    }
  }
}
// Bounded wait used on the abort path only (about 0.1 s, no error reporting).
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_test(bar, parity) && clock64() - t0 < (1ll << 28)) {}
}
// 3-D tiled TMA load (x = K element, y = row, z = slice) into shared memory,
// completing `bytes` of the barrier's transaction count.
__device__ __forceinline__ void tma_load3(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier once every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
// 32 TMEM lanes (this warp's quarter) x W consecutive 32-bit columns; the
// registers are valid after tc_wait_ld
template <int W>
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&r)[W]) {
  static_assert(W == 2 || W == 4 || W == 8, "widths used by the epilogue");
  if constexpr (W == 2) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
  } else if constexpr (W == 4) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
  } else {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr));
  }
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

struct TcMaps {
  CUtensorMap a, bre, bim;   // (Kp, rows, S) BF16 slices, box (64, 128 | BN, 1), 128-byte swizzle
  CUtensorMap bmag;          // guarded: (Kp, n, 1) magnitudes of B, box (64, 32 | 16, 1)
};

template <bool WIDE, int BITS, int BN, bool FULL = false, bool GUARD = false>   // BITS: slice width, 0 = a.bits
__global__ void __launch_bounds__(tc_threads(BN), 1) k_oz_gemm_tc(const __grid_constant__ TcMaps maps, OzArgs a,
                                                             int* err) {
  constexpr int TC_B_HALF = tc_b_half(BN), TC_B_TILE = 2 * TC_B_HALF, NSTACK = tc_nstack(BN), CPW = 4 * BN / tc_epi_warps(BN);
  constexpr int PC = CPW < 4 ? CPW : 4, MAG = GUARD ? tc_mag_cols(BN) : 0;
  if (a.active && *a.active == 0) return;   // flush with nothing pending (uniform over the grid)
  extern __shared__ uint8_t tc_smem_raw[];
  const uint32_t raw = smem_u32(tc_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* basep = tc_smem_raw + (base - raw);
  const int S = FULL ? OZ_FP64_S : a.S, SA = S + (GUARD ? 1 : 0);   // A slices per K block
  const uint32_t sB = base, strideB = (uint32_t)tc_b_bytes(S, BN, MAG);   // [2] S B tiles (and the magnitudes)
  const uint32_t sA = base + 2u * strideB;                      // [TC_ARING] A tiles of 16 KB
  const uint32_t sBar = sA + TC_ARING * TC_A_TILE;              // barriers
  uint64_t* bars = reinterpret_cast<uint64_t*>(basep + (sBar - base));
  // barrier slots: full_b 0-1, empty_b 2-3, full_a FA.., empty_a EA.., a chunk's
  // accumulators final ACC, TMEM drained by the epilogue TE, MMA thread done DONE
  constexpr int FA = 4, EA = FA + TC_ARING, ACC = EA + TC_ARING, TE = ACC + 1, DONE = TE + 1, NBAR = DONE + 1;
  auto bar = [&](int k) { return sBar + 8u * k; };
  volatile int* s_abort = reinterpret_cast<volatile int*>(bars + NBAR);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + NBAR + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // output tiles, taken persistently: CTA x handles tiles x, x + gridDim.x, ...
  // (tile t: row block t / tiles_x, column block t % tiles_x)
  const int tiles_x = (a.n + BN - 1) / BN;
  const int ntiles = tiles_x * ((a.m + TC_BM - 1) / TC_BM);
  const int my_tiles = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int nkb_all = (a.Kp + TC_BK - 1) / TC_BK;
  const int kb0 = a.kchunk ? (int)blockIdx.z * a.kchunk : 0;
  const int kb1 = a.kchunk ? min(nkb_all, kb0 + a.kchunk) : nkb_all;
  const int nkb = kb1 > kb0 ? kb1 - kb0 : 0;
  const int U = my_tiles * nkb;                                 // K blocks this CTA streams, all tiles
  auto tile_of = [&](int tt, int& i0, int& j0) {
    const int t = (int)blockIdx.x + tt * (int)gridDim.x;
    i0 = (t / tiles_x) * TC_BM;
    j0 = (t % tiles_x) * BN;
  };
  const uint32_t ncols = tc_tmem_cols(S * 2 * BN + MAG);

  if (threadIdx.x == 0) {
    for (int k = 0; k < 2; ++k) { mbar_init(bar(k), 1); mbar_init(bar(2 + k), 1); }
    for (int k = 0; k < TC_ARING; ++k) { mbar_init(bar(FA + k), 1); mbar_init(bar(EA + k), 1); }
    mbar_init(bar(ACC), 1);
    mbar_init(bar(TE), tc_epi_warps(BN));
    mbar_init(bar(DONE), 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  int armed[2 + TC_ARING] = {};   // producer: phases armed per full barrier (B 0-1, A from 2)
  if (warp == 0) {
    // ---- TMA producer: K block u = (tile u / nkb, kb0 + u % nkb) ----
    if (lane == 0 && U > 0) {
      int a_use = 0;
      int b_next = 0;   // next K block whose B slices are to be issued
      // the B slices of block u into buffer u & 1, once it is free;
      // block = false only tests whether it is free
      auto issue_b = [&](int u, bool block) -> bool {
        const int bb = u & 1;
        const uint32_t parity = ((u >> 1) & 1) ^ 1;
        if (block ? !mbar_wait(bar(2 + bb), parity, err, s_abort) : !mbar_test(bar(2 + bb), parity)) return false;
        armed[bb] = u + 1;
        int i0, j0;
        tile_of(u / nkb, i0, j0);
        const int kb = kb0 + u % nkb;
        mbar_expect_tx(bar(bb), strideB);
        if constexpr (GUARD)
          tma_load3(sB + (uint32_t)bb * strideB + (uint32_t)S * TC_B_TILE, &maps.bmag, bar(bb), kb * TC_BK, j0, 0);
        for (int q = 0; q < S; ++q) {
          const uint32_t dst = sB + (uint32_t)bb * strideB + (uint32_t)q * TC_B_TILE;
          tma_load3(dst, &maps.bre, bar(bb), kb * TC_BK, j0, q);
          tma_load3(dst + TC_B_HALF, &maps.bim, bar(bb), kb * TC_BK, j0, q);
        }
        return true;
      };
      for (int u = 0; u < U && !*s_abort; ++u) {
        if (b_next == u) {
          if (!issue_b(u, true)) break;
          ++b_next;
        }
        int i0, j0;
        tile_of(u / nkb, i0, j0);
        const int kb = kb0 + u % nkb;
        for (int p = 0; p < SA; ++p, ++a_use) {
          // the next block's B as early as its buffer is free (without waiting)
          if (b_next == u + 1 && u + 1 < U && issue_b(u + 1, false)) ++b_next;
          const int slot = a_use % TC_ARING;
          if (!mbar_wait(bar(EA + slot), ((a_use / TC_ARING) & 1) ^ 1, err, s_abort)) break;
          armed[2 + slot] = a_use / TC_ARING + 1;
          mbar_expect_tx(bar(FA + slot), (uint32_t)TC_A_TILE);
          tma_load3(sA + (uint32_t)slot * TC_A_TILE, &maps.a, bar(FA + slot), kb * TC_BK, i0, p);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    if (lane == 0) {
      int a_use = 0;
      int vt = 0;   // chunks finished so far (over all tiles)
      for (int u = 0; u < U && !*s_abort; ++u) {
        const int kbi = u % nkb, bb = u & 1;
        const bool chunk0 = kbi % a.kexact == 0;   // first K block of an exact accumulation
        if (chunk0 && u > 0) {
          // the epilogue has read the previous chunk's accumulators out of TMEM
          if (!mbar_wait(bar(TE), (vt - 1) & 1, err, s_abort)) break;
          tc_fence_after();
        }
        if (!mbar_wait(bar(bb), (u >> 1) & 1, err, s_abort)) break;
        tc_fence_after();
        bool ok = true;
        for (int p = 0; p < SA; ++p, ++a_use) {
          const int slot = a_use % TC_ARING;
          if (!mbar_wait(bar(FA + slot), (a_use / TC_ARING) & 1, err, s_abort)) { ok = false; break; }
          tc_fence_after();
          const uint64_t ad = tc_desc(sA + (uint32_t)slot * TC_A_TILE);
          if (GUARD && p == S) {   // the magnitudes, summed over the whole tile
            const uint64_t bd = tc_desc(sB + (uint32_t)bb * strideB + (uint32_t)S * TC_B_TILE);
#pragma unroll
            for (int kk = 0; kk < TC_BK / 16; ++kk)
              tc_mma(tmem + (uint32_t)(S * 2 * BN), ad + 2u * kk, bd + 2u * kk, tc_idesc(MAG > 0 ? MAG : 16),
                     (kbi == 0 && kk == 0) ? 0u : 1u);
          }
          for (int q = 0; q + p < S; q += NSTACK) {
            // pairs (p + 1, q + 1 ..) belong to groups t = p + q + 2 ..: accumulator columns from (p + q) * 64
            const int cnt = min(NSTACK, S - p - q);
            const uint64_t bd = tc_desc(sB + (uint32_t)bb * strideB + (uint32_t)q * TC_B_TILE);
            const uint32_t d = tmem + (uint32_t)(p + q) * (2 * BN);
            const uint32_t idesc = tc_idesc(2 * BN * cnt);
#pragma unroll
            for (int kk = 0; kk < TC_BK / 16; ++kk)
              tc_mma(d, ad + 2u * kk, bd + 2u * kk, idesc, (chunk0 && p == 0 && kk == 0) ? 0u : 1u);
          }
          tc_commit(bar(EA + slot));  // A slot free once these MMAs have read it
        }
        tc_commit(bar(2 + bb));       // B buffer free
        if (!ok) break;
        if ((kbi + 1) % a.kexact == 0 || kbi == nkb - 1) {
          tc_commit(bar(ACC));        // this chunk's accumulators final
          ++vt;
        }
      }
      tc_commit(bar(DONE));           // every MMA issued has completed (the abort path waits on it)
    }
  } else if (U > 0) {
    // ---- epilogue: warps from 2 on, in each TMEM lane quarter (warp % 4); warp w
    //      takes the CPW columns of group (w - 2) / 4 of each tile, chunk by chunk ----
    const int quarter = warp & 3;
    const int cg = (warp - 2) >> 2;
    const uint32_t tq = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(CPW * cg);
    const int bits = BITS ? BITS : a.bits;
    const int sh = oz_wide_shift(bits), e0 = -bits * (S + 1);
    const int ghi = WIDE ? S - oz_wide_groups() : S;   // groups of the (high) word
    const bool plain = oz_plain(a), neg = a.alpha.x < 0.0;
    const bool simple = plain && !a.rs && !a.cs;   // alpha = +-1, beta in {0, 1}, no extra scalings
    const int nch = (nkb + a.kexact - 1) / a.kexact;
    for (int tt = 0; tt < my_tiles; ++tt) {
      int i0, j0;
      tile_of(tt, i0, j0);
      j0 += CPW * cg;
      const int row = i0 + 32 * quarter + lane;
      long long ar[CPW], ai[CPW], lr[WIDE ? CPW : 1], li[WIDE ? CPW : 1];   // the tile's sums
#pragma unroll
      for (int c = 0; c < CPW; ++c) { ar[c] = 0; ai[c] = 0; }
#pragma unroll
      for (int c = 0; c < (WIDE ? CPW : 1); ++c) { lr[c] = 0; li[c] = 0; }
      uint32_t mg[CPW] = {};   // the magnitude sums
      bool have = true;
      // several chunks only in the full form: the mixed form's widths take all of K at once
      for (int ch = 0; ch < (FULL ? nch : 1); ++ch) {
        const bool waited = mbar_wait(bar(ACC), (FULL ? tt * nch + ch : tt) & 1, err, s_abort);
        // tcgen05.ld is warp-collective: the decision must be uniform over the warp
        have = __all_sync(0xffffffffu, waited && !*s_abort);
        if (!have) break;
        __syncwarp();
        tc_fence_after();
#pragma unroll 1
        for (int g = 0; g < ghi; ++g) {
          uint32_t ur[CPW], ui[CPW];
          tc_ld<CPW>(tq + (uint32_t)(g * 2 * BN), ur);
          tc_ld<CPW>(tq + (uint32_t)(g * 2 * BN + BN), ui);
          tc_wait_ld();
#pragma unroll
          for (int c = 0; c < CPW; ++c) {
            ar[c] += (long long)__float2int_rn(__uint_as_float(ur[c])) << (bits * (ghi - 1 - g));
            ai[c] += (long long)__float2int_rn(__uint_as_float(ui[c])) << (bits * (ghi - 1 - g));
          }
        }
        if constexpr (WIDE) {
#pragma unroll 1
          for (int g = ghi; g < S; ++g) {
            uint32_t ur[CPW], ui[CPW];
            tc_ld<CPW>(tq + (uint32_t)(g * 2 * BN), ur);
            tc_ld<CPW>(tq + (uint32_t)(g * 2 * BN + BN), ui);
            tc_wait_ld();
#pragma unroll
            for (int c = 0; c < CPW; ++c) {
              lr[c] += (long long)__float2int_rn(__uint_as_float(ur[c])) << (bits * (S - 1 - g));
              li[c] += (long long)__float2int_rn(__uint_as_float(ui[c])) << (bits * (S - 1 - g));
            }
          }
        }
        if (GUARD && ch == nch - 1) {
          tc_ld<CPW>(tq + (uint32_t)(S * 2 * BN), mg);
          tc_wait_ld();
        }
        // this chunk's accumulators are all in registers: TMEM may take the next chunk
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(TE));
      }
      if (!have) break;
      if (!FULL && row >= a.m) continue;
      if (a.acc) {
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          if (j0 + c >= a.n || row >= a.m) continue;
          unsigned long long* qa = a.acc + (GUARD ? 5 : WIDE ? 4 : 2) * ((size_t)(j0 + c) * a.m + row);
          if constexpr (GUARD) atomicAdd(qa + 4, __float2ull_ru(__uint_as_float(mg[c]) * 0x1p40f));
          atomicAdd(qa, (unsigned long long)ar[c]);
          if constexpr (WIDE) {
            atomicAdd(qa + 1, (unsigned long long)lr[c]);
            atomicAdd(qa + 2, (unsigned long long)ai[c]);
            atomicAdd(qa + 3, (unsigned long long)li[c]);
          } else {
            atomicAdd(qa + 1, (unsigned long long)ai[c]);
          }
        }
        continue;
      }
      const cplx beta = a.beta;
      const bool rd = beta.x != 0.0 || beta.y != 0.0;
      const bool rowin = !FULL || row < a.m;
      unsigned need = 0;   // full form: columns that the slices do not carry
      // the scale sA sB 2^-bits(S+1) is a power of two: the value is the exact
      // integer rounded once with that exponent on the integer units (GB300
      // issues FP64 at a small fraction of its integer rate); the FP64
      // operations left are the extra scalings and the addition of the old C.
      // Passes of 4 columns (2 at BN = 8), the loads (scales, old C) of a pass
      // issued before its first store.
      const int e_row = rowin ? oz_expo(a.sA[row]) + e0 : 0;
#pragma unroll
      for (int hh = 0; hh < CPW; hh += PC) {
        cplx cold[PC];
        int e_col[PC];
        bool window = true;
#pragma unroll
        for (int c = 0; c < PC; ++c) {
          const int col = j0 + hh + c;
          const bool in = col < a.n && rowin;
          cold[c] = rd && in ? a.C[(size_t)col * a.ldc + row] : cmake(0.0, 0.0);
          e_col[c] = in ? oz_expo(a.sB[col]) + e_row : 0;
          window = window && oz_window(e_col[c]);
        }
        if (window && simple) {
#pragma unroll
          for (int c = 0; c < PC; ++c) {
            if (j0 + hh + c >= a.n || !rowin) continue;
            cplx v = cmake(oz_value<WIDE>(ar[hh + c], lr[WIDE ? hh + c : 0], sh, e_col[c], true),
                           oz_value<WIDE>(ai[hh + c], li[WIDE ? hh + c : 0], sh, e_col[c], true));
            if (neg) v = cmake(-v.x, -v.y);
            if (rd) v = cadd(cold[c], v);
            if (FULL && a.A && !oz_carried<GUARD>(a, __uint_as_float(mg[hh + c]), e_col[c] - e0, v, rd)) {
              need |= 1u << (hh + c);
              continue;
            }
            a.C[(size_t)(j0 + hh + c) * a.ldc + row] = v;
          }
        } else {
#pragma unroll
          for (int c = 0; c < PC; ++c) {
            const int col = j0 + hh + c;
            if (col >= a.n || !rowin) continue;
            cplx v = cmake(oz_value<WIDE>(ar[hh + c], lr[WIDE ? hh + c : 0], sh, e_col[c], window),
                           oz_value<WIDE>(ai[hh + c], li[WIDE ? hh + c : 0], sh, e_col[c], window));
            if (e_col[c] > OZ_EXPO_NAN / 2) v = cmake(nan(""), nan(""));
            if constexpr (FULL) v = oz_scale2(a, v, row, col);
            else if (a.rs || a.cs) v = cscale(v, (a.rs ? a.rs[row] : 1.0) * (a.cs ? a.cs[col] : 1.0));
            v = oz_combine(a, beta, v, cold[c], plain);
            if (FULL && a.A && !oz_carried<GUARD>(a, __uint_as_float(mg[hh + c]), e_col[c] - e0, v, false)) {
              need |= 1u << (hh + c);
              continue;
            }
            a.C[(size_t)col * a.ldc + row] = v;
          }
        }
      }
      if constexpr (FULL) {
        if (__any_sync(0xffffffffu, need != 0u))
#pragma unroll 1
          for (int c = 0; c < CPW; ++c) oz_dot(a, row, j0 + c, (need >> c & 1u) != 0u);
      }
    }
  }
  // ---- teardown: on an abort, let issued copies and MMAs finish (bounded) ----
  __syncthreads();
  if (*s_abort) {
    if (threadIdx.x == 32) {
      mbar_drain(bar(DONE), 0);  // the MMA thread's final commit: every MMA it issued has completed
    } else if (threadIdx.x == 0) {
      for (int k = 0; k < 2; ++k)
        if (armed[k]) mbar_drain(bar(k), (armed[k] - 1) & 1);
      for (int k = 0; k < TC_ARING; ++k)
        if (armed[2 + k]) mbar_drain(bar(FA + k), (armed[2 + k] - 1) & 1);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

}  // namespace

// Slice count S and width `bits` of the mixed form's products with inner
// dimension K and a target of target_bits mantissa bits: the smallest S whose
// widest exact width in one accumulation over all of K, bits = floor((24 -
// log2(K' S)) / 2) (at most 8, the BF16 integer range), reaches the target.
// Returns false when no S <= 8 does (the product keeps one TMEM accumulator
// of 64 columns per group: 8 groups fill the 512 columns).
bool ozaki_plan(int K, int target_bits, int* S_out, int* bits_out) {
  const double kp = 2.0 * ((K + 15) / 16 * 16);
  for (int S = 2; S <= TC_MAXS; ++S) {
    int bits = (int)std::floor((24.0 - std::log2(kp * S)) / 2.0);
    if (bits > 8) bits = 8;
    if (bits < 1) return false;
    if (S * bits >= target_bits) {
      *S_out = S;
      *bits_out = bits;
      return true;
    }
  }
  return false;
}

// K blocks of 64 per exact accumulation: 64 blocks (S + 2) 2^(2 bits - 2) <= 2^24
static int oz_chunk_blocks(int S, int bits) {
  return (int)((1ll << (24 - 2 * bits + 2)) / (S + 2) / TC_BK);
}

static bool oz_full(int S) { return S == OZ_FP64_S; }

OzSlices ozaki_slices(void* scratch, int m, int n, int K, int S, int bits, bool guard) {
  const int Kpad = (K + 15) / 16 * 16;
  const size_t Kp = 2 * (size_t)Kpad;
  OzSlices o;
  o.As = reinterpret_cast<__nv_bfloat16*>(scratch);
  o.Bre = o.As + (size_t)(S + (guard ? 1 : 0)) * m * Kp;
  o.Bim = o.Bre + (size_t)S * n * Kp;
  __nv_bfloat16* end = o.Bim + (size_t)S * n * Kp;
  o.Bmag = guard ? end : nullptr;
  o.sA = reinterpret_cast<double*>(end + (guard ? (size_t)n * Kp : 0));
  o.sB = o.sA + m;
  o.m = m; o.n = n; o.Kpad = Kpad; o.S = S; o.bits = bits;
  return o;
}

// Scratch: As S*m*Kp, Bre/Bim S*n*Kp bf16 (full form: (m + n)*Kp more for the magnitudes), scales m + n doubles.
size_t ozaki_scratch_bytes(int m, int n, int K, int S) {
  const size_t Kpad = ((size_t)K + 15) / 16 * 16;
  const size_t Kp = 2 * Kpad;
  return (S * ((size_t)m + 2 * (size_t)n) + (oz_full(S) ? (size_t)m + n : 0)) * Kp * sizeof(__nv_bfloat16) +
         ((size_t)m + n) * sizeof(double) + 256;
}

// cuTensorMapEncodeTiled from the driver, looked up once (no link against libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// SMs of the current device, looked up once per device.
static int sm_count_of_current_device() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) return 148;
    cached[dev] = v;
  }
  return cached[dev];
}

// BF16 slices (Kp, rows, S), K contiguous: box of 64 K elements (128 bytes,
// the swizzle span) x box_rows rows x 1 slice, 128-byte swizzle.
static bool encode_slices(CUtensorMap* map, const __nv_bfloat16* base, size_t Kp, int rows, int S, int box_rows) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)S};
  cuuint64_t strides[2] = {(cuuint64_t)(Kp * 2), (cuuint64_t)(Kp * 2 * rows)};
  cuuint32_t box[3] = {(cuuint32_t)TC_BK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
static cudaError_t launch_tc(int which, dim3 grid, int S, cudaStream_t st, const TcMaps& maps, const OzArgs& a,
                             int* err) {
  static SmemLimit limits[6];
  void (*const kernels_tc[6])(TcMaps, OzArgs, int*) = {k_oz_gemm_tc<false, 5, BN>, k_oz_gemm_tc<false, 6, BN>,
                                                       k_oz_gemm_tc<false, 7, BN>, k_oz_gemm_tc<false, 0, BN>,
                                                       k_oz_gemm_tc<true, 7, BN>,  k_oz_gemm_tc<true, 0, BN>};
  if (cudaError_t e = limits[which].raise((const void*)kernels_tc[which], (int)tc_smem_bytes(TC_MAXS, BN, 0));
      e != cudaSuccess)
    return e;
  kernels_tc[which]<<<grid, tc_threads(BN), tc_smem_bytes(S, BN, 0), st>>>(maps, a, err);
  return cudaSuccess;
}
template <int BN, bool GUARD>
static cudaError_t launch_tc_full(dim3 grid, cudaStream_t st, const TcMaps& maps, const OzArgs& a, int* err) {
  static SmemLimit limit;
  constexpr size_t smem = tc_smem_bytes(OZ_FP64_S, BN, GUARD ? tc_mag_cols(BN) : 0);
  void (*const fn)(TcMaps, OzArgs, int*) = k_oz_gemm_tc<true, OZ_FP64_BITS, BN, true, GUARD>;
  if (cudaError_t e = limit.raise((const void*)fn, (int)smem); e != cudaSuccess) return e;
  fn<<<grid, tc_threads(BN), smem, st>>>(maps, a, err);
  return cudaSuccess;
}
template <bool GUARD>
static cudaError_t launch_tc_full(int bn, dim3 grid, cudaStream_t st, const TcMaps& maps, const OzArgs& a, int* err) {
  return bn == 8    ? launch_tc_full<8, GUARD>(grid, st, maps, a, err)
         : bn == 16 ? launch_tc_full<16, GUARD>(grid, st, maps, a, err)
                    : launch_tc_full<TC_BN_FULL, GUARD>(grid, st, maps, a, err);
}

// Complex columns BN of a tile: as narrow as keeps all tiles (times the layers of
// split K) in one wave.  A tile's time is 3 us until its first MMA, the MMAs and
// 8 us of epilogue at BN = 32, and the last two shrink with BN; A, in
// exchange, is read by more CTAs, which a long K does not repay beyond one wave.
// Flush of 16 sites, us, BN = 32 / 16 / 8: n = 256 23 / 19 / 17, n = 400 (8 slices of
// 7 bits) 27 / 22 / 24, n = 576 20 / 19 / 21, n = 1024 31 / 34 / 44; product of n = 256
// 35 / 31 / 39, of n = 576 105 / 131 / 178.
static int tc_width(int m, int nn, int layers, int ksteps, int sms, int widest) {
  const int rows = (m + TC_BM - 1) / TC_BM, most = ksteps <= 4 ? sms + sms / 4 : sms;
  for (int bn = 8; bn < widest; bn *= 2)
    if (rows * ((nn + bn - 1) / bn) * layers <= most) return bn;
  return widest;
}

cudaError_t launch_ozaki_zgemm(int m, int nn, int k, char opA, char opB, cplx alpha, const cplx* A, int lda,
                               const cplx* B, int ldb, cplx beta, cplx* C, int ldc, const double* rowscale,
                               const double* colscale, int S, int bits, void* scratch, size_t scratch_bytes,
                               unsigned long long* acc, size_t acc_bytes, cudaStream_t st, const int* active,
                               int splitk, int* kernels, int* err, bool persistent, bool presliced, bool guard) {
  const bool full = oz_full(S);
  if (S < 1 || (S > TC_MAXS && !full) || bits < 1 || bits > 8 || !err) return cudaErrorInvalidValue;
  if (full && bits != OZ_FP64_BITS) return cudaErrorInvalidValue;
  guard = guard && full;
  if ((guard && presliced) || (active && !presliced)) return cudaErrorInvalidValue;
  const int Kpad = (k + 15) / 16 * 16;
  const size_t Kp = 2 * (size_t)Kpad;
  if (ozaki_scratch_bytes(m, nn, k, S) > scratch_bytes) return cudaErrorInvalidValue;
  const OzSlices sl = ozaki_slices(scratch, m, nn, k, S, bits, guard);
  if (!presliced) {   // otherwise the slices are already in scratch (cut by the local updates; A and B are null)
    const size_t smem = (size_t)SPLIT_V * (k + 1) * sizeof(cplx);
    static SmemLimit limit_split;
    if (cudaError_t e = limit_split.raise((const void*)k_oz_split, SPLIT_V * (1024 + 1) * (int)sizeof(cplx));
        e != cudaSuccess)
      return e;
    const int vecs = m > nn ? m : nn;
    k_oz_split<<<dim3((vecs + SPLIT_V - 1) / SPLIT_V, 2), 64 * SPLIT_V, smem, st>>>(A, lda, opA, B, ldb, opB, k, sl);
  }
  OzArgs a;
  a.A = presliced ? nullptr : A; a.B = B; a.lda = lda; a.ldb = ldb; a.k = k; a.opA = opA; a.opB = opB;
  a.theta = guard ? (float)std::ldexp(std::sqrt(2.0 * k), -8) : 0.0f;
  a.theta_e = guard ? (int)std::ceil(std::log2((double)a.theta)) : 0;
  a.sA = sl.sA; a.sB = sl.sB;
  a.m = m; a.n = nn; a.Kp = (int)Kp; a.S = S; a.bits = bits;
  a.alpha = alpha; a.beta = beta; a.C = C; a.ldc = ldc; a.rs = rowscale; a.cs = colscale; a.active = active;
  // |sum_t g_t 2^{bits (S+1-t)}| < 2^{24 + bits (S-1) + 1}: one 64-bit word below 2^62, else two words
  const bool wide = 24 + bits * (S - 1) > 61;
  a.kexact = oz_chunk_blocks(S, bits);
  a.kchunk = 0;
  a.acc = nullptr;
  // persistent CTAs: one per SM (each holds the whole TMEM), every CTA takes
  // tiles x, x + grid, ... and overlaps a tile's epilogue with the next tile's
  // MMAs; otherwise one CTA per tile (chains sharing the GPU: short CTAs let
  // the other chains' kernels in between)
  const int sms = sm_count_of_current_device();
  const int ksteps = (int)((Kp + TC_BK - 1) / TC_BK);
  if (a.kexact < (full ? 1 : ksteps)) return cudaErrorInvalidValue;
  int layers = 1;
  if (splitk > 1 && !active && ksteps > 1 && acc &&
      (size_t)m * nn * (guard ? 5 : wide ? 4 : 2) * sizeof(unsigned long long) <= acc_bytes) {
    // split K over blockIdx.z: exact 64-bit integer partial sums in acc, which
    // is zero between products (zeroed at allocation, re-zeroed by the finaliser)
    if (splitk > ksteps) splitk = ksteps;
    a.kchunk = (ksteps + splitk - 1) / splitk;
    layers = (ksteps + a.kchunk - 1) / a.kchunk;
    a.acc = acc;
  }
  const int widest = full ? TC_BN_FULL : TC_BN;
  const int bn = persistent ? tc_width(m, nn, layers, ksteps, sms, widest) : widest;
  const int ntiles = ((nn + bn - 1) / bn) * ((m + TC_BM - 1) / TC_BM);
  const dim3 grid(persistent && ntiles > sms ? sms : ntiles, 1, layers);
  if (kernels) *kernels = (a.acc ? 3 : 2) - (presliced ? 1 : 0);
  {
    TcMaps maps;
    if (!encode_slices(&maps.a, sl.As, Kp, m, S + (guard ? 1 : 0), TC_BM) ||
        !encode_slices(&maps.bre, sl.Bre, Kp, nn, S, bn) || !encode_slices(&maps.bim, sl.Bim, Kp, nn, S, bn))
      return cudaErrorInvalidValue;
    if (guard && !encode_slices(&maps.bmag, sl.Bmag, Kp, nn, 1, tc_mag_cols(bn))) return cudaErrorInvalidValue;
    // the widths of the default targets are compiled in: 5, 6, 7 (40 bits, by K), 7 in two words (56 bits)
    const int which = wide ? (bits == 7 ? 4 : 5) : bits == 5 ? 0 : bits == 6 ? 1 : bits == 7 ? 2 : 3;
    const cudaError_t e = full      ? (guard ? launch_tc_full<true>(bn, grid, st, maps, a, err)
                                             : launch_tc_full<false>(bn, grid, st, maps, a, err))
                        : bn == 32 ? launch_tc<32>(which, grid, S, st, maps, a, err)
                        : bn == 16 ? launch_tc<16>(which, grid, S, st, maps, a, err)
                                   : launch_tc<8>(which, grid, S, st, maps, a, err);
    if (e != cudaSuccess) return e;
  }
  if (a.acc) {
    const size_t total = (size_t)m * nn;
    const int blocks = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    if (guard) k_oz_finalize<true, true, true><<<blocks, 256, 0, st>>>(a);
    else if (full) k_oz_finalize<true, true><<<blocks, 256, 0, st>>>(a);
    else if (wide) k_oz_finalize<true><<<blocks, 256, 0, st>>>(a);
    else k_oz_finalize<false><<<blocks, 256, 0, st>>>(a);
  }
  return cudaGetLastError();
}
