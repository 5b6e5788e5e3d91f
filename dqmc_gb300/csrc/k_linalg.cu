// Dense complex FP64 linear algebra for the UDT stabilisation.
//
// Reference: src/linalg.jl:20-39 (decompose_udt! = LAPACK zgeqp3 + zungqr),
// src/stack.jl:338-369 (calculate_greens) and src/stack.jl:278-313
// (add_slice_sequence_*).  The column-pivoted Householder QR restates the
// published LAPACK algorithm (zgeqp3/zlaqp2: pivot = first column of maximal
// partial norm, zlarfg reflector, column-norm downdating with the
// sqrt(eps) recomputation guard).  Columns are never moved: a logical ->
// physical order array replaces LAPACK's column swaps, so the triangular
// factor comes out directly in the un-permuted ("T = R[:, invperm(p)]")
// layout that the UDT decomposition needs.
#include <cfloat>
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace {

// ---------------------------------------------------------------------------
// GEMM: C = alpha * diag(rs) * op(A) * op(B) * diag(cs) + beta * C
// ---------------------------------------------------------------------------
constexpr int GB_M = 64, GB_N = 64, GB_K = 8;

__device__ __forceinline__ cplx load_op(const cplx* X, int ld, int r, int c, int rows, int cols, char op) {
  // element (r, c) of op(X); op(X) has shape rows x cols
  if (r >= rows || c >= cols) return cmake(0.0, 0.0);
  if (op == 'N') return X[(size_t)c * ld + r];
  cplx v = X[(size_t)r * ld + c];
  return op == 'C' ? cconj(v) : v;
}

__global__ void __launch_bounds__(256) k_zgemm(int m, int nn, int k, char opA, char opB, cplx alpha,
                                              const cplx* __restrict__ A, int lda, const cplx* __restrict__ B,
                                              int ldb, cplx beta, cplx* __restrict__ C, int ldc,
                                              const double* __restrict__ rs, const double* __restrict__ cs) {
  __shared__ cplx sA[GB_K][GB_M + 1];
  __shared__ cplx sB[GB_K][GB_N + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int i0 = blockIdx.y * GB_M, j0 = blockIdx.x * GB_N;
  cplx acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = cmake(0.0, 0.0);
  for (int k0 = 0; k0 < k; k0 += GB_K) {
    for (int e = threadIdx.x; e < GB_M * GB_K; e += 256) {
      int kk, ii;
      if (opA == 'N') { ii = e % GB_M; kk = e / GB_M; } else { kk = e % GB_K; ii = e / GB_K; }
      sA[kk][ii] = load_op(A, lda, i0 + ii, k0 + kk, m, k, opA);
      int jj, kb;
      if (opB == 'N') { kb = e % GB_K; jj = e / GB_K; } else { jj = e % GB_N; kb = e / GB_N; }
      sB[kb][jj] = load_op(B, ldb, k0 + kb, j0 + jj, k, nn, opB);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GB_K; ++kk) {
      cplx av[4], bv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) av[a] = sA[kk][ty + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) bv[b] = sB[kk][tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = cfma(av[a], bv[b], acc[a][b]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    int i = i0 + ty + 16 * a;
    if (i >= m) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      int j = j0 + tx + 16 * b;
      if (j >= nn) continue;
      cplx v = acc[a][b];
      if (rs) v = cscale(v, rs[i]);
      if (cs) v = cscale(v, cs[j]);
      v = cmul(alpha, v);
      cplx* cp = &C[(size_t)j * ldc + i];
      if (beta.x != 0.0 || beta.y != 0.0) v = cfma(beta, *cp, v);
      *cp = v;
    }
  }
}

// ---------------------------------------------------------------------------
// warp / block reductions
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ cplx warp_sum(cplx v) { return cmake(warp_sum(v.x), warp_sum(v.y)); }

// block-wide sum, deterministic (fixed tree); all threads get the result.
__device__ double block_sum(double v, double* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  double t = 0.0;
  for (int q = 0; q < nw; ++q) t += scratch[q];
  return t;
}

// ---------------------------------------------------------------------------
// column-pivoted QR (cooperative, one grid barrier per column step)
// ---------------------------------------------------------------------------
constexpr int QR_THREADS = 256;
constexpr int QR_WARPS = QR_THREADS / 32;              // the last one is the reflector warp
constexpr int QR_REFL_WORDS = 10;                      // beta, tau, scal in 32-bit halves under the step's tag
constexpr int QR_MAXT = 32;   // elements per lane of one column (n <= 1024)
constexpr int CAND_PER_LANE = 8;   // per-CTA pivot candidates read per lane: grids of at most 256 CTAs

// Candidate of the next pivot: the CTA-local maximum of the partial norms
// and its logical position (ties: smaller position, as LAPACK's idamax).
// Norms are >= +0, so their bit patterns order like their values: the
// comparison runs on the integer units, not the FP64 unit.
__device__ __forceinline__ bool cand_better(double v, int q, double bv, int bq) {
  const long long a = __double_as_longlong(v), b = __double_as_longlong(bv);
  return a > b || (a == b && q < bq);
}

// Complex warp sum with five FP64 adds: after one exchange the low half of
// the warp reduces the real parts and the high half the imaginary parts.
__device__ __forceinline__ cplx warp_sum_c(cplx v) {
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 16;
  double keep = hi ? v.y : v.x;
  const double send = hi ? v.x : v.y;
  keep += __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
  return cmake(__shfl_sync(0xffffffffu, keep, 0), __shfl_sync(0xffffffffu, keep, 16));
}

// a -= c v over the column slots of one lane (c = f at r = k, f scal below,
// v_k = 1), stored back; with TAIL the squared norm of the updated rows > k.
template <bool TAIL>
__device__ __forceinline__ double qr_update_column(cplx (&x)[QR_MAXT], cplx* __restrict__ col, const cplx* v, int k,
                                                   int n, int nq, int lane, cplx f, cplx fs) {
  double tp = 0.0;
#pragma unroll
  for (int q = 0; q < QR_MAXT; ++q) {
    if (q >= nq) break;
    const int r = k + lane + 32 * q;
    if (r < n) {
      // four fused multiply-adds per element
      const cplx vr = r == k ? cmake(1.0, 0.0) : v[r];
      const cplx c = r == k ? f : fs;
      x[q] = cmake(fma(-c.x, vr.x, fma(c.y, vr.y, x[q].x)), fma(-c.x, vr.y, fma(-c.y, vr.x, x[q].y)));
      col[r] = x[q];
      if (TAIL && r > k) tp = fma(x[q].x, x[q].x, fma(x[q].y, x[q].y, tp));
    }
  }
  return tp;
}

// sum_{r > k} conj(x_r) a_r over one lane's slots (loads the column into x)
__device__ __forceinline__ cplx qr_load_dot(cplx (&x)[QR_MAXT], const cplx* __restrict__ col, const cplx* v, int k,
                                            int n, int nq, int lane) {
  cplx sp = cmake(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < QR_MAXT; ++q) {
    if (q >= nq) break;
    const int r = k + lane + 32 * q;
    x[q] = cmake(0.0, 0.0);
    if (r < n) {
      x[q] = ldcg_c(&col[r]);
      if (r > k) sp = cfma_conj(v[r], x[q], sp);
    }
  }
  return warp_sum_c(sp);
}

// loads one lane's slots of a column into x (as qr_load_dot, without the dot)
__device__ __forceinline__ void qr_load(cplx (&x)[QR_MAXT], const cplx* __restrict__ col, int k, int n, int nq,
                                        int lane) {
#pragma unroll
  for (int q = 0; q < QR_MAXT; ++q) {
    if (q >= nq) break;
    const int r = k + lane + 32 * q;
    x[q] = r < n ? ldcg_c(&col[r]) : cmake(0.0, 0.0);
  }
}

// sum_{r > k} conj(x_r) a_r over one lane's slots already in x (the order of qr_load_dot)
__device__ __forceinline__ cplx qr_dot(const cplx (&x)[QR_MAXT], const cplx* v, int k, int n, int nq, int lane) {
  cplx sp = cmake(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < QR_MAXT; ++q) {
    if (q >= nq) break;
    const int r = k + lane + 32 * q;
    if (r < n && r > k) sp = cfma_conj(v[r], x[q], sp);
  }
  return warp_sum_c(sp);
}

// One column step after the dot product s0 = sum_{r>k} conj(x_r) a_r:
// a -= tau^H (v^H a) v with v = (1, scal x_{k+1..n}), then the partial norm
// downdate of zlaqp2 with stored reciprocals (vn1, vn2 at [j], 1/vn1, 1/vn2
// at [n + j]); returns the new partial norm.
__device__ __forceinline__ double qr_finish_column(cplx (&x)[QR_MAXT], cplx* __restrict__ col, const cplx* v, int k,
                                                   int n, int nq, int lane, int j, cplx s0, cplx ctau, cplx scal,
                                                   const QRWork& w, double tol3z) {
  const double vn1 = __ldcg(&w.vn1[j]), vn2 = __ldcg(&w.vn2[j]);
  const double inv1 = __ldcg(&w.vn1[n + j]), inv2 = __ldcg(&w.vn2[n + j]);
  // v^H a = a_k + conj(scal) s0
  const cplx ak = cmake(__shfl_sync(0xffffffffu, x[0].x, 0), __shfl_sync(0xffffffffu, x[0].y, 0));
  const cplx s = cfma_conj(scal, s0, ak);
  const cplx f = cmul(ctau, s);     // a_k -= f
  const cplx fs = cmul(f, scal);    // a_r -= f scal x_r, r > k
  // zlaqp2: temp = max(0, 1 - (|a_k|/vn1)^2), temp2 = temp (vn1/vn2)^2;
  // recompute the norm when temp2 <= sqrt(eps), else vn1 *= sqrt(temp)
  double vn1_new = vn1, inv1_new = inv1;
  bool recompute = false;
  if (vn1 != 0.0) {
    const cplx xk = csub(ak, f);
    double temp = 1.0 - (cabs2(xk) * inv1) * inv1;
    temp = temp > 0.0 ? temp : 0.0;
    const double r2 = vn1 * inv2;
    if (temp * r2 * r2 <= tol3z) {
      recompute = true;
    } else {
      const double rs = rsqrt(temp);
      vn1_new = vn1 * temp * rs;
      inv1_new = inv1 * rs;
    }
  }
  if (recompute) {
    const double tail = warp_sum(qr_update_column<true>(x, col, v, k, n, nq, lane, f, fs));
    vn1_new = (k < n - 1) ? sqrt(tail) : 0.0;
    inv1_new = vn1_new > 0.0 ? 1.0 / vn1_new : 0.0;
    if (lane == 0) { w.vn2[j] = vn1_new; w.vn2[n + j] = inv1_new; }
  } else {
    qr_update_column<false>(x, col, v, k, n, nq, lane, f, fs);
  }
  if (lane == 0 && vn1 != 0.0) { w.vn1[j] = vn1_new; w.vn1[n + j] = inv1_new; }
  return vn1_new;
}

// Column step k: the pivot column p (the first of maximal partial norm) gives the
// reflector; every other column is updated and its norm downdated, one warp per
// column, the remaining columns dealt round-robin over the CTAs.  One grid
// barrier per step.  The reflector's scalars are a chain of a square root and two
// divisions (about 5000 cycles with the norm), which every CTA runs ahead of time
// for its own candidate while the grid barrier is under way, on its last warp
// (which takes columns only once the others all have one).  The chosen one's
// owner has published them by the time the others have read the column and
// formed their first dot products.  Bound: FP64 issue while more than a few
// hundred columns remain, then the latency of barrier, pivot column and norm
// downdate.  Per sequence of calls, ms, formed after the barrier -> ahead:
// n = 64 1.70 -> 1.53, 144 8.0 -> 7.4, 256 14.9 -> 14.4, 1024 52.6 -> 51.8.
__global__ void __launch_bounds__(QR_THREADS, 1) k_qrp(cplx* __restrict__ A, int n, int kend, QRWork w) {
  unsigned epoch = 0;
  GridBarrierExit bar_exit(w.bar);
  extern __shared__ double smem_qr[];
  cplx* v = reinterpret_cast<cplx*>(smem_qr);         // (n) pivot column: a_k at k, unscaled x below
  int* order = reinterpret_cast<int*>(v + n);         // (n) logical -> physical
  __shared__ double red[QR_WARPS], nsum[QR_WARPS];
  __shared__ int redi[QR_WARPS], redj[QR_WARPS];
  __shared__ cplx s_tau, s_scal;
  __shared__ int s_ok, s_wc, s_rok;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int warps = QR_WARPS, CT = 32 * (QR_WARPS - 1);   // CT: threads of the other warps
  const bool refl_warp = wid == warps - 1;
  const int gwarp = blockIdx.x * warps + wid, nwarps = gridDim.x * warps;
  const double tol3z = sqrt(DBL_EPSILON);

  for (int q = threadIdx.x; q < n; q += blockDim.x) order[q] = q;
  // initial column norms (zgeqp3: vn1 = vn2 = ||A(:, j)||) and the first candidates
  double cbest = 0.0;
  int cbq = n, cbj = 0;
  for (int j = gwarp; j < n; j += nwarps) {
    double s = 0.0;
    for (int r = lane; r < n; r += 32) s += cabs2(A[(size_t)j * n + r]);
    s = warp_sum(s);
    const double nv = sqrt(s), iv = nv > 0.0 ? 1.0 / nv : 0.0;
    if (lane == 0) { w.vn1[j] = nv; w.vn2[j] = nv; w.vn1[n + j] = iv; w.vn2[n + j] = iv; }
    if (cand_better(nv, j, cbest, cbq)) { cbest = nv; cbq = j; cbj = j; }
  }
  for (int e = threadIdx.x; e < 2 * QR_REFL_WORDS; e += blockDim.x)   // this CTA's reflector slots are empty
    w.refl[((size_t)(e / QR_REFL_WORDS) * gridDim.x + blockIdx.x) * QR_REFL_WORDS + e % QR_REFL_WORDS] = 0ull;

  const int chunk = (n + gridDim.x - 1) / gridDim.x;   // rows of V written by this CTA
  for (int k = 0; k < kend; ++k) {
    const int rem = n - k - 1;
    const int nq = (n - k + 31) >> 5;   // warp-uniform: no FP64 work on fully masked slots
    const int t_first = blockIdx.x + gridDim.x * wid;
    const int par = k & 1;
    // ---- this CTA's candidate of step k (lane 0 of each warp holds its best) ----
    if (lane == 0) { red[wid] = cbest; redi[wid] = cbq; redj[wid] = cbj; }
    __syncthreads();   // the columns of step k - 1 are stored
    double cb = red[0];
    int cq = redi[0], cj = redj[0];
#pragma unroll
    for (int q = 1; q < warps; ++q)
      if (cand_better(red[q], redi[q], cb, cq)) { cb = red[q]; cq = redi[q]; cj = redj[q]; }
    ++epoch;
    if (wid == 0) {
      // ---- arrive at the grid barrier with the candidate, wait, choose the pivot ----
      int ok = 1;
      if (lane == 0) {
        w.cand_v[par * gridDim.x + blockIdx.x] = cb;
        w.cand_q[par * gridDim.x + blockIdx.x] = cq;
        __threadfence();
        atomicAdd(&w.bar->count, 1u);
        long long spins = 0;
        while (ld_acquire_u32(&w.bar->count) < epoch * gridDim.x) {
          if ((++spins & 1023) == 0) {
            if (spins > (1ll << 26)) { atomicOr(w.err, 2); ok = 0; break; }
            if (*(volatile int*)w.err & 2) { ok = 0; break; }
          }
        }
        __threadfence();
        s_ok = ok;
      }
      __syncwarp();
    } else if (cq < n) {
      // ---- the reflector of this CTA's candidate (zlarfg): partial squared norms
      //      of its column below row k, summed as 8 warps with rows 256 apart per
      //      thread; the reflector warp takes the first warp's share as well ----
      cplx x0 = cmake(0.0, 0.0);
      for (int wp = refl_warp ? 0 : wid; wp < warps; wp += refl_warp ? warps - 1 : warps) {
        double xn2 = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int r = k + 32 * wp + lane + u * QR_THREADS;
          if (r < n) {
            const cplx x = ldcg_c(&A[(size_t)cj * n + r]);
            if (u == 0 && wp == 0) x0 = x;
            if (r > k) xn2 = fma(x.x, x.x, fma(x.y, x.y, xn2));
          }
        }
        xn2 = warp_sum(xn2);
        if (lane == 0) nsum[wp] = xn2;
      }
      __syncwarp();
      if (!refl_warp) {
        asm volatile("bar.arrive 1, 224;" ::: "memory");
      } else {
        asm volatile("bar.sync 1, 224;" ::: "memory");
        double t = lane < warps ? nsum[lane] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);   // warps <= 8
        const cplx alpha = cmake(__shfl_sync(0xffffffffu, x0.x, 0), __shfl_sync(0xffffffffu, x0.y, 0));
        t = __shfl_sync(0xffffffffu, t, 0);
        double beta;
        cplx tau, scal;
        if (t == 0.0 && alpha.y == 0.0) {
          tau = cmake(0.0, 0.0);
          beta = alpha.x;
          scal = cmake(0.0, 0.0);
        } else {
          const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + t);
          beta = alpha.x >= 0.0 ? -nrm : nrm;
          const double rb = 1.0 / beta;
          tau = cmake((beta - alpha.x) * rb, -alpha.y * rb);
          // scal = 1 / (alpha - beta), formed on (alpha - beta) / nrm (modulus in [1, 2])
          const double an = fabs(rb);
          const cplx dd = cmake((alpha.x - beta) * an, alpha.y * an);
          const double rd = an / (dd.x * dd.x + dd.y * dd.y);
          scal = cmake(dd.x * rd, -dd.y * rd);
        }
        // words of 32 bits under the step's tag validate themselves
        if (lane < QR_REFL_WORDS) {
          const int c = lane >> 1;
          const double val = c == 0 ? beta : c == 1 ? tau.x : c == 2 ? tau.y : c == 3 ? scal.x : scal.y;
          const unsigned half = lane & 1 ? (unsigned)__double2loint(val) : (unsigned)__double2hiint(val);
          unsigned long long* o = w.refl + ((size_t)par * gridDim.x + blockIdx.x) * QR_REFL_WORDS + lane;
          asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(o), "l"((unsigned long long)(k + 1) << 32 | half)
                       : "memory");
        }
      }
    }
    // ---- column warps: the barrier is passed; first columns read while the pivot
    //      is chosen (read again if the exchange moves another column there) ----
    cplx x[QR_MAXT];
    int j_pre = -1;
    if (!refl_warp) {
      asm volatile("bar.sync 2, 224;" ::: "memory");
      if (s_ok) {
        if (t_first < rem) {
          j_pre = order[k + 1 + t_first];
          qr_load(x, A + (size_t)j_pre * n, k, n, nq, lane);
        }
        // best of the per-CTA candidates (first position of maximal norm), warp 0
        if (wid == 0) {
          // all candidate loads in flight at once (grid <= 32 * CAND_PER_LANE), then the compares
          double cvv[CAND_PER_LANE];
          int cqq[CAND_PER_LANE];
#pragma unroll
          for (int u = 0; u < CAND_PER_LANE; ++u) {
            const int c = lane + 32 * u;
            cvv[u] = 0.0;
            cqq[u] = n;
            if (c < (int)gridDim.x) {
              cvv[u] = __ldcg(&w.cand_v[par * gridDim.x + c]);
              cqq[u] = __ldcg(&w.cand_q[par * gridDim.x + c]);
            }
          }
          double best = 0.0;
          int bestq = n, bc = 0;
#pragma unroll
          for (int u = 0; u < CAND_PER_LANE; ++u)
            if (cand_better(cvv[u], cqq[u], best, bestq)) { best = cvv[u]; bestq = cqq[u]; bc = lane + 32 * u; }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            double ob = __shfl_xor_sync(0xffffffffu, best, o);
            int oq = __shfl_xor_sync(0xffffffffu, bestq, o), oc = __shfl_xor_sync(0xffffffffu, bc, o);
            if (cand_better(ob, oq, best, bestq)) { best = ob; bestq = oq; bc = oc; }
          }
          if (lane == 0) {
            const bool none = bestq < k || bestq >= n;   // NaN in every remaining column: keep the order
            s_wc = none ? -1 : bc;
            if (none) bestq = k;
            int t = order[k]; order[k] = order[bestq]; order[bestq] = t;
          }
          __syncwarp();
        }
      }
    }
    __syncthreads();
    if (!s_ok) return;
    // ---- the reflector warp fetches the chosen reflector; the column warps read
    //      the pivot column and form their first dot products (which need neither) ----
    cplx s_first = cmake(0.0, 0.0);
    int j_first = -1;
    if (refl_warp) {
      const int wc = s_wc;
      const unsigned long long* src = w.refl + ((size_t)par * gridDim.x + max(wc, 0)) * QR_REFL_WORDS + lane;
      unsigned long long word = 0x7FF8000000000000ull >> (lane & 1 ? 0 : 32);   // halves of a NaN: the reflector of NaN columns
      bool here = wc < 0;
      for (long long spins = 0; !here && spins < (1ll << 22); ++spins) {
        if (lane < QR_REFL_WORDS)
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(word) : "l"(src) : "memory");
        here = __all_sync(0xffffffffu, lane >= QR_REFL_WORDS || (unsigned)(word >> 32) == (unsigned)(k + 1));
      }
      if (!here && lane == 0) atomicOr(w.err, 2);
      double f[5];
#pragma unroll
      for (int c = 0; c < 5; ++c)
        f[c] = __hiloint2double((int)__shfl_sync(0xffffffffu, (unsigned)word, 2 * c),
                                (int)__shfl_sync(0xffffffffu, (unsigned)word, 2 * c + 1));
      if (lane == 0) {
        s_tau = cmake(f[1], f[2]);
        s_scal = cmake(f[3], f[4]);
        s_rok = here ? 1 : 0;
        if (blockIdx.x == 0) { w.tau[k] = cmake(f[1], f[2]); w.beta[k] = f[0]; }
      }
    } else {
      const int p = order[k];
#pragma unroll
      for (int u = 0; u < 5; ++u) {   // n <= 1024 < 5 CT
        const int r = k + threadIdx.x + u * CT;
        if (r < n) v[r] = ldcg_c(&A[(size_t)p * n + r]);
      }
      asm volatile("bar.sync 2, 224;" ::: "memory");
      if (t_first < rem) {
        j_first = order[k + 1 + t_first];
        if (j_first != j_pre) qr_load(x, A + (size_t)j_first * n, k, n, nq, lane);
        s_first = qr_dot(x, v, k, n, nq, lane);
      }
    }
    __syncthreads();   // tau, scal visible
    if (!s_rok) return;
    const cplx ctau = cconj(s_tau), scal = s_scal;
    cbest = 0.0;
    cbq = n;
    cbj = 0;
    // rows of V written by this CTA: v = (1, scal x_{k+1..n}), zero above k
    for (int r = blockIdx.x * chunk + threadIdx.x; r < n && r < (blockIdx.x + 1) * chunk; r += blockDim.x)
      w.V[(size_t)k * n + r] = r < k ? cmake(0.0, 0.0) : (r == k ? cmake(1.0, 0.0) : cmul(v[r], scal));
    // ---- apply H_k^H to the remaining columns, downdate their norms ----
    // remaining logical positions k+1..n-1 are dealt round-robin over the CTAs
    // first, so every SM keeps an equal share of the columns as k grows
    if (j_first >= 0) {
      const double nv = qr_finish_column(x, A + (size_t)j_first * n, v, k, n, nq, lane, j_first, s_first, ctau, scal,
                                         w, tol3z);
      if (lane == 0 && cand_better(nv, k + 1 + t_first, cbest, cbq)) {
        cbest = nv; cbq = k + 1 + t_first; cbj = j_first;
      }
    }
    // further columns of this warp (more columns than warps), and the reflector
    // warp's share when it has one
    for (int t = refl_warp ? t_first : t_first + gridDim.x * warps; t < rem; t += gridDim.x * warps) {
      const int qpos = k + 1 + t;
      const int j = order[qpos];
      cplx* col = A + (size_t)j * n;
      const cplx s0 = qr_load_dot(x, col, v, k, n, nq, lane);
      const double nv = qr_finish_column(x, col, v, k, n, nq, lane, j, s0, ctau, scal, w, tol3z);
      if (lane == 0 && cand_better(nv, qpos, cbest, cbq)) { cbest = nv; cbq = qpos; cbj = j; }
    }
  }
  if (blockIdx.x == 0)
    for (int q = threadIdx.x; q < n; q += blockDim.x) w.order[q] = order[q];
}

// Block j of the compact-WY form of Q = H_0 ... H_{n-1}: Vb (m x b, m = n - jb,
// leading dimension m) = rows jb.. of reflector columns jb..jb+b; a reflector
// with tau = 0 is the identity and is stored as v = 0 with tau' = 1, so that
// T^-1 = diag(1/tau') + striu(Vb^H Vb) stays valid.  trd = tau'.
__global__ void k_wy_prep(const cplx* __restrict__ V, const cplx* __restrict__ tau, int n, int jb, int b,
                          cplx* __restrict__ Vb, cplx* __restrict__ trd) {
  const int m = n - jb;
  const size_t total = (size_t)m * b;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(e / m), r = (int)(e - (size_t)c * m);
    const cplx t = tau[jb + c];
    const bool ident = t.x == 0.0 && t.y == 0.0;
    Vb[e] = ident ? cmake(0.0, 0.0) : V[(size_t)(jb + c) * n + jb + r];
    if (r == 0) trd[c] = ident ? cmake(1.0, 0.0) : t;
  }
}

// C = A + B over count complex entries
__global__ void k_add(const cplx* __restrict__ A, const cplx* __restrict__ B, cplx* __restrict__ C, size_t count) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x)
    C[e] = cadd(A[e], B[e]);
}

__global__ void k_iota(int* __restrict__ p, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = i;
}

// D-scale separation helpers: s[0..n) = 1/max(Dl,1), s[n..2n) = min(Dl,1),
// s[2n..3n) = 1/max(Dr,1), s[3n..4n) = min(Dr,1)
__global__ void k_split_scales(const double* __restrict__ Dl, const double* __restrict__ Dr, int n,
                               double* __restrict__ s) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double l = Dl[i], r = Dr[i];
    s[i] = 1.0 / (l > 1.0 ? l : 1.0);
    s[n + i] = l < 1.0 ? l : 1.0;
    s[2 * n + i] = 1.0 / (r > 1.0 ? r : 1.0);
    s[3 * n + i] = r < 1.0 ? r : 1.0;
  }
}

// out[0] = sum_i log|u_i| + log max(Dl_i, 1) + log max(Dr_i, 1)  (single CTA)
__global__ void k_lu_logdet(const cplx* __restrict__ udiag, const double* __restrict__ Dl,
                            const double* __restrict__ Dr, int n, double* out) {
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double l = Dl[i], r = Dr[i];
    s += 0.5 * log(cabs2(udiag[i])) + log(l > 1.0 ? l : 1.0) + log(r > 1.0 ? r : 1.0);
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[0] = s;
}

// ---------------------------------------------------------------------------
// column-pivoted QR with the columns in registers (cooperative)
// ---------------------------------------------------------------------------
// Steps k0 .. n - 1 of k_qrp when at most four columns per SM remain: one column
// per warp and sub-partition, from the launch's start to its pivot step, so no
// step loads or stores columns, and a CTA's chain from one pivot to the next
// passes no grid barrier.  Per step:
//   warps 0-3   a column each: its norm as the CTA's bid for the next pivot; the
//               update of the step before (beside the exchange), which the bidding
//               column publishes; then the dot product and the norm;
//   warp 4      publishes the CTA's bid, polls all CTAs', picks the pivot;
//   warps 4-11  fetch the pivot column, sum its squares, write rows of V;
//   warp 5      the reflector's scalars (in every CTA: a second way through L2
//               costs more than the sum and the chain of a root and two divisions).
// A norm that has to be recomputed (the guard of zlaqp2) needs the update and a
// further pass.  It is below 2^-12 of its last exact value, so the CTA bids with
// its best exact norm if that is larger, else with the bound, and the pivot is
// waited for only where a bound turns out to be the best bid.
// What CTAs publish validates itself: a bid is one 16-byte word with the step's
// tag, columns are 32-bit halves under the tag.  Buffers alternate by step:
// nobody publishes step k + 2 before all have published step k + 1, which they
// do after reading everything of step k.
// Rows stay with their lanes (row base + 32 q + lane), and the sums over a
// column rotate to the lanes that k_qrp has them in: same terms in the same
// order, so both kernels give the same bits.
// Bound: latency; a step of n = 144 is update, the way through L2, squares and
// scalars (6000 cycles) and the norm downdate (2000).  From n = 400 on the passes
// over a column at one FP64 instruction per 64 cycles and sub-partition take over.
// Per sequence of calls, ms, k_qrp -> this: n = 64 1.53 -> 1.24, 144 7.4 -> 5.9,
// 256 14.4 -> 10.8, 400 31.7 -> 24.4, 576 41.4 -> 36.0, 1024 (the last 608 columns)
// 51.8 -> 49.6.
constexpr int QC_COLS = 4, QC_HELP = 8;
constexpr int QC_THREADS = 32 * (QC_COLS + QC_HELP);
// named barriers
constexpr int QC_B_BIDS = 1, QC_B_NORMS = 2, QC_B_PIVOT = 3, QC_B_TAU = 4, QC_B_EXACT = 5, QC_B_COL = 8, QC_B_COLTAU = 12;
constexpr int QC_SLOTS = 5;                     // candidates polled per lane: grids of at most 160 CTAs
constexpr int QC_POLLS = 1 << 20;               // bound of every wait (about a second)
constexpr long long QC_NONE = -0x7FFFFFFFFFFFFFFFll - 1;   // key of a CTA without columns

__device__ __forceinline__ void qc_sync(int id, int warps) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(32 * warps) : "memory");
}
__device__ __forceinline__ void qc_arrive(int id, int warps) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(32 * warps) : "memory");
}
__device__ __forceinline__ void qc_store16(unsigned long long* p, unsigned long long a, unsigned long long b) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p), "l"(a),
               "l"(b)
               : "memory");
}
__device__ __forceinline__ void qc_load16(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ unsigned long long qc_word(unsigned tag, int half) {
  return (unsigned long long)tag << 32 | (unsigned)half;
}
// a == b ? x : y, kept a select (as an indexed read the columns would live in local memory)
__device__ __forceinline__ double qc_select(int a, int b, double x, double y) {
  double r;
  asm("{\n .reg .pred p;\n setp.eq.s32 p, %1, %2;\n selp.f64 %0, %3, %4, p;\n}\n" : "=d"(r) : "r"(a), "r"(b), "d"(x), "d"(y));
  return r;
}
// norms order like their bit patterns; a NaN with its sign set comes last
__device__ __forceinline__ long long qc_key(double norm) {
  const long long b = __double_as_longlong(norm);
  return b < 0 ? -1 : b;
}

template <int NQ>   // rows from k0's group of 32 on, in groups of 32
__global__ void __launch_bounds__(QC_THREADS, 1) k_qr_cols(cplx* __restrict__ A, int n, int k0, QRWork w) {
  extern __shared__ double smem_qc[];
  const int base = k0 & ~31, rows = n - base;
  cplx* vbuf = reinterpret_cast<cplx*>(smem_qc);   // (2, rows) pivot columns, by step parity
  __shared__ long long s_key[2][QC_COLS], s_exact[2][QC_COLS];
  __shared__ int s_pos[2][QC_COLS], s_phys[2][QC_COLS], s_def[2][QC_COLS];
  __shared__ int s_win[2][3];                      // pivot: CTA, logical position, column
  __shared__ double s_norm[QC_HELP];
  __shared__ cplx s_tau[2], s_scal[2];
  __shared__ int s_abort;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, G = gridDim.x;
  const unsigned run = *(volatile unsigned*)w.run + 1u;   // tags differ from those of earlier launches and of k_qrp
  if (threadIdx.x == 0) s_abort = 0;
  __syncthreads();
  volatile int* abort = &s_abort;
  unsigned long long* slot = w.slots;                               // (2, to, from, 2)
  unsigned long long* cols = w.cols;                                // (2, G, rows, 4)
  auto give_up = [&] {   // nothing is waited for any more; the results are void
    if (!*abort) { atomicOr(w.err, DQMC_KERR_BARRIER_TIMEOUT); *abort = 1; }
  };
  // The CTA's candidate among the columns with an exact norm, in key; open: a
  // deferred column (s_def, key a bound) may be better, bound its bound.
  auto cta_best = [&](int par, long long& key, bool& open, long long& bound) {
    int c = 0;
    key = QC_NONE;
    bound = QC_NONE;
#pragma unroll
    for (int q = 0; q < QC_COLS; ++q) {
      const long long kq = s_key[par][q];
      if (s_def[par][q]) {
        if (kq > bound) bound = kq;
      } else if (kq > key || (kq == key && s_pos[par][q] < s_pos[par][c])) {
        key = kq;
        c = q;
      }
    }
    open = bound != QC_NONE && bound >= key;
    return c;
  };
  auto cta_best_exact = [&](int par, long long& key) {
    int c = 0;
    key = s_exact[par][0];
#pragma unroll
    for (int q = 1; q < QC_COLS; ++q)
      if (s_exact[par][q] > key || (s_exact[par][q] == key && s_pos[par][q] < s_pos[par][c])) {
        key = s_exact[par][q];
        c = q;
      }
    return c;
  };

  // warp 4: this CTA's bid to all, theirs, the pivot of step k
  auto pick_pivot = [&](int k) {
    const int par = k & 1;
    const unsigned tag = run * 2048u + (unsigned)k + 1u;
    qc_sync(QC_B_BIDS, QC_COLS + 1);
    long long key, bound;
    bool open;
    int c = cta_best(par, key, open, bound);
    // a mailbox per receiver: polled by one CTA each, where common slots would
    // serialise 150 pollers in a few L2 slices
    auto publish = [&](long long kq, unsigned meta) {
      for (int e = lane; e < G; e += 32)
        qc_store16(slot + (((size_t)par * G + e) * G + blockIdx.x) * 2, (unsigned long long)kq,
                   (unsigned long long)tag << 32 | meta);
    };
    if (open) {
      publish(bound, 0x80000000u);
      qc_sync(QC_B_EXACT, QC_COLS + 1);
      c = cta_best_exact(par, key);
    }
    publish(key, (unsigned)(s_pos[par][c] << 16 | s_phys[par][c]));
    const unsigned long long* sl = slot + ((size_t)par * G + blockIdx.x) * G * 2;
    unsigned long long kk[QC_SLOTS], mm[QC_SLOTS];
    unsigned have = 0;
#pragma unroll
    for (int u = 0; u < QC_SLOTS; ++u)
      if (lane + 32 * u >= G) { have |= 1u << u; kk[u] = (unsigned long long)QC_NONE; mm[u] = 0xFFFFFFFFull; }
    for (int it = 0;; ++it) {
#pragma unroll
      for (int u = 0; u < QC_SLOTS; ++u)
        if (!(have >> u & 1)) qc_load16(sl + 2 * (lane + 32 * u), kk[u], mm[u]);
#pragma unroll
      for (int u = 0; u < QC_SLOTS; ++u)
        if ((unsigned)(mm[u] >> 32) == tag) have |= 1u << u;
      if (__all_sync(0xffffffffu, have == (1u << QC_SLOTS) - 1)) break;
      if (it >= QC_POLLS || ((it & 1023) == 1023 && (*abort || (*(volatile int*)w.err & DQMC_KERR_BARRIER_TIMEOUT)))) {
        give_up();
        break;
      }
    }
    __syncwarp();
    // the best; a bound that is best (m < 0, before equal exact norms) is waited for
    long long bk;
    int bm, bc;
    for (int it = 0;; ++it) {
      bk = QC_NONE;
      bm = 0x7FFFFFFF;
      bc = 0;
#pragma unroll
      for (int u = 0; u < QC_SLOTS; ++u) {
        const int m = (int)(unsigned)mm[u];
        if (lane + 32 * u < G && ((long long)kk[u] > bk || ((long long)kk[u] == bk && m < bm))) {
          bk = (long long)kk[u]; bm = m; bc = lane + 32 * u;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const long long ok = __shfl_xor_sync(0xffffffffu, bk, o);
        const int om = __shfl_xor_sync(0xffffffffu, bm, o), oc = __shfl_xor_sync(0xffffffffu, bc, o);
        if (ok > bk || (ok == bk && om < bm)) { bk = ok; bm = om; bc = oc; }
      }
      if (bm >= 0) break;
      if (it >= QC_POLLS || ((it & 1023) == 1023 && (*abort || (*(volatile int*)w.err & DQMC_KERR_BARRIER_TIMEOUT)))) {
        give_up();
        break;
      }
#pragma unroll
      for (int u = 0; u < QC_SLOTS; ++u)
        if (lane + 32 * u < G && (int)(unsigned)mm[u] < 0) qc_load16(sl + 2 * (lane + 32 * u), kk[u], mm[u]);
    }
    if (lane == 0) {
      s_win[par][0] = bc;
      s_win[par][1] = (bm >> 16) & 0x7FFF;
      s_win[par][2] = min(bm & 0xFFFF, n - 1);
    }
    __syncwarp();
  };

  if (wid < QC_COLS) {
    // ---- a column ----
    const int i0 = blockIdx.x + G * wid;
    bool active = i0 < n - k0;
    int pos = k0 + i0, phys = 0;
    cplx x[NQ];
    double vn1 = 0.0, vn2 = 0.0, inv1 = 0.0, inv2 = 0.0;
    if (active) {
      phys = k0 ? __ldcg(&w.order[pos]) : pos;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int r = base + lane + 32 * q;
        x[q] = r < n ? ldcg_c(&A[(size_t)phys * n + r]) : cmake(0.0, 0.0);
      }
      if (k0) {
        vn1 = __ldcg(&w.vn1[phys]); vn2 = __ldcg(&w.vn2[phys]);
        inv1 = __ldcg(&w.vn1[n + phys]); inv2 = __ldcg(&w.vn2[n + phys]);
      } else {
        double s = 0.0;
        for (int r = lane; r < n; r += 32) s += cabs2(A[(size_t)phys * n + r]);
        s = warp_sum(s);
        vn1 = sqrt(s);
        inv1 = vn1 > 0.0 ? 1.0 / vn1 : 0.0;
        vn2 = vn1;
        inv2 = inv1;
      }
    }
    const double tol3z = sqrt(DBL_EPSILON);
    bool pending = false, deferred = false;   // the update by the step before; its norm too
    cplx f = cmake(0.0, 0.0), fs = cmake(0.0, 0.0);
    // x -= c v of step k (c = f at r = k, fs below, v_k = 1); TAIL: squares below row k
    // pub: the new rows below k go to this CTA's published column of step k + 1
    auto publish = [&](int k, int q) {
      const unsigned tag = run * 2048u + (unsigned)k + 1u;
      unsigned long long* p = cols + (((size_t)(k & 1) * G + blockIdx.x) * rows + 32 * q + lane) * 4;
      asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(qc_word(tag, __double2hiint(x[q].x))),
                   "l"(qc_word(tag, __double2loint(x[q].x)))
                   : "memory");
      asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p + 2),
                   "l"(qc_word(tag, __double2hiint(x[q].y))), "l"(qc_word(tag, __double2loint(x[q].y)))
                   : "memory");
    };
    auto update = [&](int k, auto tail, bool pub) {
      const cplx* v = vbuf + (size_t)(k & 1) * rows;
      double tp = 0.0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        if (base + 32 * q + 31 < k || base + 32 * q >= n) continue;   // warp-uniform
        const int r = base + lane + 32 * q;
        if (r >= k && r < n) {
          const cplx vr = r == k ? cmake(1.0, 0.0) : v[r - base];
          const cplx c = r == k ? f : fs;
          x[q] = cmake(fma(-c.x, vr.x, fma(c.y, vr.y, x[q].x)), fma(-c.x, vr.y, fma(-c.y, vr.x, x[q].y)));
          if (decltype(tail)::value && r > k) tp = fma(x[q].x, x[q].x, fma(x[q].y, x[q].y, tp));
          if (pub && r > k) publish(k + 1, q);
        }
      }
      return tp;
    };
    for (int k = k0; k < n; ++k) {
      const int par = k & 1, d = k - base;
      const unsigned tag = run * 2048u + (unsigned)k + 1u;
      if (lane == 0) {
        // a deferred norm is below vn2 sqrt(tol3z): twice that as a power of two
        s_key[par][wid] = !active ? QC_NONE : qc_key(deferred ? vn2 * 0x1p-12 : vn1);
        s_def[par][wid] = deferred ? 1 : 0;
        s_pos[par][wid] = pos;
        s_phys[par][wid] = phys;
      }
      qc_sync(QC_B_BIDS, QC_COLS + 1);
      long long best, bound;
      bool open;
      int cw = cta_best(par, best, open, bound);
      const bool early = active && !open && cw == wid;   // this column is the CTA's bid
      if (deferred) {
        const double tp = update(k - 1, std::true_type{}, false);
        const double tail = warp_sum(__shfl_sync(0xffffffffu, tp, (lane + d - 1) & 31));
        vn1 = sqrt(tail);   // k - 1 < n - 1
        inv1 = vn1 > 0.0 ? 1.0 / vn1 : 0.0;
        vn2 = vn1;
        inv2 = inv1;
      } else if (pending) {
        update(k - 1, std::false_type{}, early);
      }
      if (open) {   // uniform over the CTA
        if (lane == 0) s_exact[par][wid] = active ? qc_key(vn1) : QC_NONE;
        qc_sync(QC_B_EXACT, QC_COLS + 1);
        cw = cta_best_exact(par, best);
      }
      if (active && cw == wid && !(early && pending)) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const int r = base + lane + 32 * q;
          if (r >= k && r < n) publish(k, q);
        }
      }
      pending = deferred = false;
      // this column's element of row k, for all lanes
      cplx ak = cmake(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        ak.x = qc_select(q, d >> 5, x[q].x, ak.x);
        ak.y = qc_select(q, d >> 5, x[q].y, ak.y);
      }
      ak = cmake(__shfl_sync(0xffffffffu, ak.x, d & 31), __shfl_sync(0xffffffffu, ak.y, d & 31));
      const int rot = (lane + d) & 31;   // the lane with k_qrp's rows k + lane, k + lane + 32, ...
      qc_sync(QC_B_COL + wid, 1 + QC_HELP);   // pivot known, its column in vbuf
      const int wpos = s_win[par][1];
      cplx s0 = cmake(0.0, 0.0);
      if (active && pos == wpos) {
        // the pivot: its rows above k are final
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const int r = base + lane + 32 * q;
          if (r < k) A[(size_t)phys * n + r] = x[q];
        }
        active = false;
      } else if (active) {
        if (pos == k) pos = wpos;
        const cplx* v = vbuf + (size_t)par * rows;
        cplx sp = cmake(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          if (base + 32 * q + 31 <= k || base + 32 * q >= n) continue;   // warp-uniform
          const int r = base + lane + 32 * q;
          if (r > k && r < n) sp = cfma_conj(v[r - base], x[q], sp);
        }
        s0 = warp_sum_c(cmake(__shfl_sync(0xffffffffu, sp.x, rot), __shfl_sync(0xffffffffu, sp.y, rot)));
      }
      qc_sync(QC_B_COLTAU + wid, 2);   // tau, scal
      if (active) {
        const cplx ctau = cconj(s_tau[par]), scal = s_scal[par];
        // v^H a = a_k + conj(scal) s0
        const cplx s = cfma_conj(scal, s0, ak);
        f = cmul(ctau, s);     // a_k -= f
        fs = cmul(f, scal);    // a_r -= f scal x_r, r > k
        pending = true;
        if (vn1 != 0.0) {      // the norm downdate of qr_finish_column
          const cplx xk = csub(ak, f);
          double temp = 1.0 - (cabs2(xk) * inv1) * inv1;
          temp = temp > 0.0 ? temp : 0.0;
          const double r2 = vn1 * inv2;
          if (temp * r2 * r2 <= tol3z) {
            deferred = true;   // recomputed beside the exchange of the next step
          } else {
            const double rs = rsqrt(temp);
            vn1 = vn1 * temp * rs;
            inv1 = inv1 * rs;
          }
        }
      }
    }
  } else {
    // ---- the other warps ----
    const int hw = wid - QC_COLS, tid = 32 * hw + lane, chunk = (n + G - 1) / G;
    constexpr int T = 32 * QC_HELP, U = (32 * NQ + T - 1) / T;
    for (int k = k0; k < n; ++k) {
      const int par = k & 1;
      const unsigned tag = run * 2048u + (unsigned)k + 1u;
      if (hw == 0) pick_pivot(k);
      qc_sync(QC_B_PIVOT, QC_HELP);
      // the pivot column; thread t holds rows k + t, k + t + 256, ... (as in k_qrp)
      cplx* v = vbuf + (size_t)par * rows;
      const unsigned long long* src = cols + ((size_t)par * G + s_win[par][0]) * rows * 4;
      unsigned have = 0;
      double xn2 = 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + tid + T * u >= n) have |= 1u << u;
      const unsigned mine = ~have;
      cplx z[U];
      for (int it = 0; have != (1u << U) - 1; ++it) {
        unsigned long long q0[U], q1[U], q2[U], q3[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (!(have >> u & 1)) {
            const unsigned long long* p = src + (size_t)(k + tid + T * u - base) * 4;
            asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(q0[u]), "=l"(q1[u]) : "l"(p) : "memory");
            asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(q2[u]), "=l"(q3[u]) : "l"(p + 2) : "memory");
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (!(have >> u & 1) && (unsigned)(q0[u] >> 32) == tag && (unsigned)(q1[u] >> 32) == tag &&
              (unsigned)(q2[u] >> 32) == tag && (unsigned)(q3[u] >> 32) == tag) {
            have |= 1u << u;
            z[u] = cmake(__hiloint2double((int)(unsigned)q0[u], (int)(unsigned)q1[u]),
                         __hiloint2double((int)(unsigned)q2[u], (int)(unsigned)q3[u]));
            v[k + tid + T * u - base] = z[u];
          }
        if (it >= QC_POLLS || ((it & 1023) == 1023 && *abort)) {
          if (have != (1u << U) - 1) give_up();
          break;
        }
      }
      __syncwarp();
#pragma unroll
      for (int c = 0; c < QC_COLS; ++c) qc_arrive(QC_B_COL + c, 1 + QC_HELP);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if ((mine & have) >> u & 1)
          if (u > 0 || tid > 0) xn2 = fma(z[u].x, z[u].x, fma(z[u].y, z[u].y, xn2));
      xn2 = warp_sum(xn2);
      if (lane == 0) s_norm[hw] = xn2;
      __syncwarp();
      if (hw != 1) {
        qc_arrive(QC_B_NORMS, QC_HELP);
      } else {
        qc_sync(QC_B_NORMS, QC_HELP);
        // zlarfg, as in k_qrp
        double t = lane < QC_HELP ? s_norm[lane] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        t = __shfl_sync(0xffffffffu, t, 0);
        const cplx alpha = v[k - base];
        double beta;
        cplx tau, scal;
        if (t == 0.0 && alpha.y == 0.0) {
          tau = cmake(0.0, 0.0);
          beta = alpha.x;
          scal = cmake(0.0, 0.0);
        } else {
          const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + t);
          beta = alpha.x >= 0.0 ? -nrm : nrm;
          const double rb = 1.0 / beta;
          tau = cmake((beta - alpha.x) * rb, -alpha.y * rb);
          const double an = fabs(rb);
          const cplx dd = cmake((alpha.x - beta) * an, alpha.y * an);
          const double rd = an / (dd.x * dd.x + dd.y * dd.y);
          scal = cmake(dd.x * rd, -dd.y * rd);
        }
        if (lane == 0) {
          s_tau[par] = tau;
          s_scal[par] = scal;
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < QC_COLS; ++c) qc_arrive(QC_B_COLTAU + c, 2);
        if (lane == 0 && blockIdx.x == 0) {
          w.tau[k] = tau;
          w.beta[k] = beta;
          w.order[k] = s_win[par][2];
        }
      }
      qc_sync(QC_B_TAU, QC_HELP);
      const cplx scal = s_scal[par];
      const int r1 = min(n, ((int)blockIdx.x + 1) * chunk);
      for (int r = blockIdx.x * chunk + tid; r < r1; r += T)
        w.V[(size_t)k * n + r] = r < k ? cmake(0.0, 0.0) : (r == k ? cmake(1.0, 0.0) : cmul(v[r - base], scal));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {   // the last CTA out counts the launch
    __threadfence();
    if (atomicAdd(&w.bar->exits, 1u) == (unsigned)G - 1) {
      w.bar->exits = 0;
      *w.run = run & 0xFFFFFu;
      __threadfence();
    }
  }
}

// T (physical layout) = D^-1 R, zero below the logical diagonal; D = |beta|.
__global__ void k_qrp_finalize(const cplx* __restrict__ A, cplx* __restrict__ T, double* __restrict__ D, int n,
                               const int* __restrict__ order, const double* __restrict__ beta) {
  extern __shared__ int pos[];   // physical -> logical
  for (int q = threadIdx.x; q < n; q += blockDim.x) pos[order[q]] = q;
  __syncthreads();
  const size_t total = (size_t)n * n;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    int j = (int)(e / n), r = (int)(e - (size_t)j * n);
    int q = pos[j];
    double d = fabs(beta[r]);
    cplx val;
    if (r < q) val = cscale(A[e], 1.0 / d);
    else if (r == q) val = cmake(beta[r] / d, 0.0);
    else val = cmake(0.0, 0.0);
    T[e] = val;
  }
  if (blockIdx.x == 0)
    for (int q = threadIdx.x; q < n; q += blockDim.x) D[q] = fabs(beta[q]);
}

// X (m x n) <- X * Q (or X * Q^H), one warp per row, row held in registers.
__global__ void __launch_bounds__(128) k_apply_q_right(cplx* __restrict__ X, int m, int n,
                                                      const cplx* __restrict__ V, const cplx* __restrict__ tau,
                                                      int conj_q) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (row >= m) return;
  cplx x[QR_MAXT];
#pragma unroll
  for (int t = 0; t < QR_MAXT; ++t) {
    int c = lane + 32 * t;
    x[t] = c < n ? X[(size_t)c * m + row] : cmake(0.0, 0.0);
  }
  for (int s = 0; s < n; ++s) {
    const int k = conj_q ? (n - 1 - s) : s;
    const cplx* vk = V + (size_t)k * n;
    cplx tk = tau[k];
    if (tk.x == 0.0 && tk.y == 0.0) continue;
    if (conj_q) tk = cconj(tk);
    // X H = X - tau (X v) v^H
    // one accumulator: the FP64 unit's issue rate, not its latency, bounds the chain
    cplx dp = cmake(0.0, 0.0);
    const int t0 = k >> 5, t1 = (n + 31) >> 5;   // warp-uniform range of slots holding columns >= k
#pragma unroll
    for (int t = 0; t < QR_MAXT; ++t) {
      if (t < t0) continue;
      if (t >= t1) break;
      int c = lane + 32 * t;
      if (c >= k && c < n) dp = cfma(x[t], __ldg(&vk[c]), dp);
    }
    cplx d = warp_sum_c(dp);
    cplx f = cmul(tk, d);
#pragma unroll
    for (int t = 0; t < QR_MAXT; ++t) {
      if (t < t0) continue;
      if (t >= t1) break;
      int c = lane + 32 * t;
      if (c >= k && c < n) {
        cplx vc = __ldg(&vk[c]);
        // x_c -= f * conj(v_c) with four fused multiply-adds
        x[t] = cmake(fma(-f.x, vc.x, fma(-f.y, vc.y, x[t].x)), fma(-f.y, vc.x, fma(f.x, vc.y, x[t].y)));
      }
    }
  }
#pragma unroll
  for (int t = 0; t < QR_MAXT; ++t) {
    int c = lane + 32 * t;
    if (c < n) X[(size_t)c * m + row] = x[t];
  }
}

// Y <- That^-1 Y, That[r, q] = T[r, order[q]] upper triangular (logical order).
// One warp per column of Y (column staged in shared memory).
__global__ void __launch_bounds__(128) k_trsm_left_upper(const cplx* __restrict__ T, const int* __restrict__ order,
                                                        cplx* __restrict__ Y, int n, int m) {
  extern __shared__ double smem_t[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int col = blockIdx.x * (blockDim.x / 32) + wid;
  if (col >= m) return;
  cplx* y = reinterpret_cast<cplx*>(smem_t) + (size_t)wid * n;
  cplx* yg = Y + (size_t)col * n;
  for (int r = lane; r < n; r += 32) y[r] = yg[r];
  __syncwarp();
  for (int q = n - 1; q >= 0; --q) {
    const cplx* tq = T + (size_t)__ldg(&order[q]) * n;
    // the unit-scaled factor of a QR has diagonal beta/|beta| = +-1: a sign, not a division
    const cplx d = __ldg(&tq[q]);
    const cplx yq = (d.y == 0.0 && fabs(d.x) == 1.0) ? cscale(y[q], d.x) : cdiv(y[q], d);
    __syncwarp();
    if (lane == 0) y[q] = yq;
    for (int r = lane; r < q; r += 32) {
      const cplx t = __ldg(&tq[r]);
      y[r] = cmake(fma(-yq.x, t.x, fma(yq.y, t.y, y[r].x)), fma(-yq.x, t.y, fma(-yq.y, t.x, y[r].y)));
    }
    __syncwarp();
  }
  for (int r = lane; r < n; r += 32) yg[r] = y[r];
}

// Diagonal-block solve of a blocked triangular solve: the b x b block of T
// at (j0, j0) (leading dimension ldT) applied to rows j0..j0+b of the m
// columns of Y (leading dimension ldY).  lower: unit lower triangular,
// forward; otherwise upper with the reciprocal diagonal rdiag[j0 + q],
// backward.  Each CTA stages the strict triangle of the block, packed by
// columns, in shared memory once (no L2 round trip inside the dependent
// column steps); each warp solves one column with its b values in registers
// (row lane + 32 i in slot i) and broadcasts y_q by shuffle.
constexpr int TRSM_DB_WARPS = 8;   // all stage the triangle; the first `warps` of them solve a column each
__device__ __forceinline__ int trsm_pack_lower(int q, int b) { return q * (b - 1) - q * (q - 1) / 2; }
__device__ __forceinline__ int trsm_pack_upper(int q) { return q * (q - 1) / 2; }

// a b with the multiply-adds spelled out (which product a compiler contracts depends on the context)
__device__ __forceinline__ cplx trsm_scale(cplx a, cplx b) {
  return cmake(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y)));
}
template <int NS>   // slots of 32 rows, b <= 32 NS
__global__ void __launch_bounds__(32 * TRSM_DB_WARPS) k_trsm_diag_block(const cplx* __restrict__ T, int ldT,
                                                                       const cplx* __restrict__ rdiag,
                                                                       cplx* __restrict__ Y, int ldY, int j0, int b,
                                                                       int m, int lower, int warps) {
  extern __shared__ double4_16a smem_tdb[];
  cplx* tp = reinterpret_cast<cplx*>(smem_tdb);   // (b (b - 1) / 2) packed strict triangle
  cplx* rd = tp + (size_t)b * (b - 1) / 2;        // (b) reciprocal diagonal (upper)
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int bb = b * b;
  for (int e0 = threadIdx.x; e0 < bb; e0 += 8 * blockDim.x) {
    cplx v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * blockDim.x;
      const int q = e / b, r = e - q * b;
      if (e < bb && (lower ? r > q : r < q)) v[u] = __ldg(&T[(size_t)(j0 + q) * ldT + j0 + r]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * blockDim.x;
      const int q = e / b, r = e - q * b;
      if (e < bb && (lower ? r > q : r < q))
        tp[lower ? trsm_pack_lower(q, b) + (r - q - 1) : trsm_pack_upper(q) + r] = v[u];
    }
  }
  if (!lower)
    for (int q = threadIdx.x; q < b; q += blockDim.x) rd[q] = __ldg(&rdiag[j0 + q]);
  __syncthreads();
  const int col = blockIdx.x * warps + wid;
  if (wid >= warps || col >= m) return;
  cplx* yg = Y + (size_t)col * ldY + j0;
  cplx y[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const int r = lane + 32 * i;
    y[i] = r < b ? yg[r] : cmake(0.0, 0.0);
  }
  auto bcast = [&](cplx v, int src) {
    return cmake(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
  };
  auto sub = [&](cplx& v, cplx yq, cplx t) {
    v = cmake(fma(-yq.x, t.x, fma(yq.y, t.y, v.x)), fma(-yq.x, t.y, fma(-yq.y, t.x, v.y)));
  };
  // Column q of the triangle is read one step ahead, and the slot that holds
  // the next step's row is updated first: the chain of a step is then a shuffle
  // and two FMAs (upper: four), about 200 cycles, and the FP64 issue of the
  // slots, 256 cycles each, is what is left.  Solves of b rows, us, before -> now:
  // b = 64 lower 34 -> 21, upper 44 -> 31 (m <= 608), upper 69 -> 44 (m = 1024);
  // b = 128 upper 89 -> 79.
  cplx t[NS], tn[NS];
  if (lower) {
    auto load = [&](int q, cplx (&o)[NS]) {
      const cplx* tq = tp + trsm_pack_lower(q, b) - q - 1;   // tq[r], r > q
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        const int r = lane + 32 * i;
        if (r > q && r < b) o[i] = tq[r];
      }
    };
    load(0, tn);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      for (int j = 0; j < 32; ++j) {
        const int q = 32 * s + j;
        if (q >= b - 1) break;
#pragma unroll
        for (int i = s; i < NS; ++i) t[i] = tn[i];
        const cplx yq = bcast(y[s], j);
        load(q + 1, tn);
#pragma unroll
        for (int i = s; i < NS; ++i) {
          const int r = lane + 32 * i;
          if (r > q && r < b) sub(y[i], yq, t[i]);
        }
      }
    }
  } else {
    auto load = [&](int q, cplx (&o)[NS]) {
      const cplx* tq = tp + trsm_pack_upper(q);   // tq[r], r < q
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        const int r = lane + 32 * i;
        if (r < q) o[i] = tq[r];
      }
    };
    load(b - 1, tn);
    cplx dn = rd[b - 1];
#pragma unroll
    for (int s = NS - 1; s >= 0; --s) {
      for (int j = 31; j >= 0; --j) {
        const int q = 32 * s + j;
        if (q >= b) continue;
#pragma unroll
        for (int i = 0; i <= s; ++i) t[i] = tn[i];
        const cplx yq = trsm_scale(bcast(y[s], j), dn);
        if (q > 0) {
          load(q - 1, tn);
          dn = rd[q - 1];
        }
#pragma unroll
        for (int i = s; i >= 0; --i) {
          const int r = lane + 32 * i;
          if (r == q) y[i] = yq;
          else if (r < q) sub(y[i], yq, t[i]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const int r = lane + 32 * i;
    if (r < b) yg[r] = y[i];
  }
}

// Y <- Y That^-1 (Y is m x n), one warp per row: z That = y, forward over columns.
__global__ void __launch_bounds__(128) k_trsm_right_upper(const cplx* __restrict__ T, const int* __restrict__ order,
                                                         cplx* __restrict__ Y, int m, int n) {
  extern __shared__ double smem_t[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int row = blockIdx.x * (blockDim.x / 32) + wid;
  if (row >= m) return;
  cplx* z = reinterpret_cast<cplx*>(smem_t) + (size_t)wid * n;
  for (int c = lane; c < n; c += 32) z[c] = Y[(size_t)c * m + row];
  __syncwarp();
  for (int q = 0; q < n; ++q) {
    const cplx* tq = T + (size_t)__ldg(&order[q]) * n;
    cplx s = cmake(0.0, 0.0);
    for (int r = lane; r < q; r += 32) s = cfma(z[r], __ldg(&tq[r]), s);
    s = warp_sum(s);
    if (lane == 0) {
      const cplx d = __ldg(&tq[q]);
      const cplx t = csub(z[q], s);
      z[q] = (d.y == 0.0 && fabs(d.x) == 1.0) ? cscale(t, d.x) : cdiv(t, d);
    }
    __syncwarp();
  }
  for (int c = lane; c < n; c += 32) Y[(size_t)c * m + row] = z[c];
}

__global__ void k_permute(const cplx* __restrict__ src, cplx* __restrict__ dst, int rows, int cols,
                          const int* __restrict__ order, int by_rows, int scatter) {
  const size_t total = (size_t)rows * cols;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    int c = (int)(e / rows), r = (int)(e - (size_t)c * rows);
    if (by_rows) {
      if (scatter) dst[(size_t)c * rows + order[r]] = src[e];
      else dst[e] = src[(size_t)c * rows + order[r]];
    } else {
      if (scatter) dst[(size_t)order[c] * rows + r] = src[e];
      else dst[e] = src[(size_t)order[c] * rows + r];
    }
  }
}

__global__ void k_add_diag(cplx* A, int n, const double* d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) A[(size_t)i * n + i].x += d[i];
}

__global__ void k_set_identity(cplx* A, int n) {
  const size_t total = (size_t)n * n;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    int c = (int)(e / n), r = (int)(e - (size_t)c * n);
    A[e] = cmake(r == c ? 1.0 : 0.0, 0.0);
  }
}

__global__ void k_scale(cplx* A, int rows, int cols, const double* rs, int inv_r, const double* cs, int inv_c) {
  const size_t total = (size_t)rows * cols;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    int c = (int)(e / rows), r = (int)(e - (size_t)c * rows);
    double f = 1.0;
    if (rs) f = inv_r ? f / rs[r] : f * rs[r];
    if (cs) f = inv_c ? f / cs[c] : f * cs[c];
    A[e] = cscale(A[e], f);
  }
}

__global__ void k_conj_transpose(const cplx* __restrict__ A, cplx* __restrict__ B, int n) {
  __shared__ cplx tile[32][33];
  int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
    int c = bx + yy, r = by + threadIdx.x;
    if (c < n && r < n) tile[yy][threadIdx.x] = A[(size_t)c * n + r];
  }
  __syncthreads();
  for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
    int c = by + yy, r = bx + threadIdx.x;   // B[r, c] = conj(A[c, r])
    if (c < n && r < n) B[(size_t)c * n + r] = cconj(tile[threadIdx.x][yy]);
  }
}

// out[0] = sum log(x)  (single CTA, deterministic)
__global__ void k_sum_log(const double* x, int n, double* out) {
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += log(x[i]);
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[0] = s;
}

__global__ void k_max_absdiff(const cplx* A, const cplx* B, size_t count, double* out) {
  __shared__ double red[32];
  double m = 0.0;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x) {
    cplx d = csub(A[e], B[e]);
    double a = sqrt(cabs2(d));
    if (!(a <= m)) m = a;   // propagates NaN
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double q = __shfl_xor_sync(0xffffffffu, m, o);
    if (!(q <= m)) m = q;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q)
      if (!(red[q] <= t)) t = red[q];
    // combine across CTAs: non-negative doubles order like their bit patterns
    unsigned long long bits = __double_as_longlong(t);
    if (t != t) bits = 0x7ff8000000000000ull;
    atomicMax(reinterpret_cast<unsigned long long*>(out), bits);
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline int grid_for(size_t total, int threads = 256, int cap = 4096) {
  size_t g = (total + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > (size_t)cap) g = cap;
  return (int)g;
}

cudaError_t launch_zgemm(int m, int nn, int k, char opA, char opB, cplx alpha, const cplx* A, int lda,
                         const cplx* B, int ldb, cplx beta, cplx* C, int ldc, const double* rowscale,
                         const double* colscale, cudaStream_t st) {
  dim3 grid((nn + GB_N - 1) / GB_N, (m + GB_M - 1) / GB_M);
  k_zgemm<<<grid, 256, 0, st>>>(m, nn, k, opA, opB, alpha, A, lda, B, ldb, beta, C, ldc, rowscale, colscale);
  return cudaGetLastError();
}

// Columns that k_qr_cols can hold (0: none) and the words of its published columns.
static int qr_resident_columns(int n, int sm_count, int max_grid) {
  int grid = sm_count < 32 * QC_SLOTS ? sm_count : 32 * QC_SLOTS;
  if (max_grid > 0 && grid > max_grid) grid = max_grid;
  const int held = QC_COLS * grid;
  if (held >= n) return n;
  return max_grid > 0 ? 0 : held;   // chains that share the GPU: all of the columns or none
}
size_t qr_column_words(int n, int sm_count) {
  const int held = qr_resident_columns(n, sm_count, 0), base = (n - held) & ~31;
  return (size_t)2 * ((held + QC_COLS - 1) / QC_COLS) * (n - base) * 4;
}

template <int NQ>
static cudaError_t launch_qr_cols(cplx* A, int n, int k0, QRWork& w, cudaStream_t st) {
  const int base = k0 & ~31, grid = (n - k0 + QC_COLS - 1) / QC_COLS;
  QRWork copy = w;
  void* args[] = {&A, &n, &k0, &copy};
  return cudaLaunchCooperativeKernel((void*)k_qr_cols<NQ>, dim3(grid), dim3(QC_THREADS), args,
                                     (size_t)2 * (n - base) * sizeof(cplx), st);
}

// The last columns, as many as the SMs hold, by k_qr_cols; k_qrp takes the steps
// before (n > 608 on 152 SMs) or, where the held ones are too few, all.
cudaError_t launch_qrp(cplx* A, int n, QRWork& w, int sm_count, cudaStream_t st, int max_grid, int* kernels) {
  if (n > 32 * QR_MAXT) return cudaErrorInvalidValue;
  int held = qr_resident_columns(n, sm_count, max_grid), kend = n - held;
  *kernels = (kend > 0 ? 1 : 0) + (held > 0 ? 1 : 0);
  if (kend > 0) {
    size_t smem = (size_t)n * (sizeof(cplx) + sizeof(int));
    static SmemLimit smem_limit;
    if (cudaError_t ea = smem_limit.raise((const void*)k_qrp, 64 * 1024); ea != cudaSuccess) return ea;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_qrp, QR_THREADS, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    int grid = sm_count;   // one CTA per SM; remaining columns are dealt round-robin over all CTAs
    if (max_grid > 0 && grid > max_grid) grid = max_grid;
    if (grid > 32 * CAND_PER_LANE) grid = 32 * CAND_PER_LANE;
    QRWork copy = w;
    void* args[] = {&A, &n, &kend, &copy};
    e = cudaLaunchCooperativeKernel((void*)k_qrp, dim3(grid), dim3(QR_THREADS), args, smem, st);
    if (e != cudaSuccess || held == 0) return e;
  }
  const int nq = (n - (kend & ~31) + 31) / 32;   // at most 21 (640 held columns)
  if (nq <= 2) return launch_qr_cols<2>(A, n, kend, w, st);
  if (nq <= 5) return launch_qr_cols<5>(A, n, kend, w, st);
  if (nq <= 8) return launch_qr_cols<8>(A, n, kend, w, st);
  if (nq <= 13) return launch_qr_cols<13>(A, n, kend, w, st);
  if (nq <= 18) return launch_qr_cols<18>(A, n, kend, w, st);
  if (nq <= 21) return launch_qr_cols<21>(A, n, kend, w, st);
  return cudaErrorInvalidValue;
}
cudaError_t launch_qrp_finalize(cplx* A, cplx* T, double* D, int n, const QRWork& w, cudaStream_t st) {
  k_qrp_finalize<<<grid_for((size_t)n * n), 256, n * sizeof(int), st>>>(A, T, D, n, w.order, w.beta);
  return cudaGetLastError();
}

cudaError_t launch_apply_q_right(cplx* X, int m, int n, const QRWork& w, bool conj_transpose_q, cudaStream_t st) {
  if (n > 32 * QR_MAXT) return cudaErrorInvalidValue;
  // one row per warp, 4 warps per CTA: up to 2 CTAs per SM at 256 registers per thread
  int rows_per_cta = 4;
  k_apply_q_right<<<(m + rows_per_cta - 1) / rows_per_cta, 128, 0, st>>>(X, m, n, w.V, w.tau,
                                                                        conj_transpose_q ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_trsm_left_upper(const cplx* T, const int* order, cplx* Y, int n, int m, cudaStream_t st) {
  size_t smem = (size_t)4 * n * sizeof(cplx);
  static SmemLimit smem_limit;
  if (cudaError_t ea = smem_limit.raise((const void*)k_trsm_left_upper, 200 * 1024); ea != cudaSuccess) return ea;
  k_trsm_left_upper<<<(m + 3) / 4, 128, smem, st>>>(T, order, Y, n, m);
  return cudaGetLastError();
}

cudaError_t launch_trsm_diag_block(const cplx* T, int ldT, const cplx* rdiag, cplx* Y, int ldY, int j0, int b, int m,
                                   bool lower, cudaStream_t st) {
  if (b < 1 || b > 128) return cudaErrorInvalidValue;
  if (!lower && !rdiag) return cudaErrorInvalidValue;
  const size_t smem = ((size_t)b * (b - 1) / 2 + b) * sizeof(cplx);
  constexpr int kMaxTdb = (int)((128 * 127 / 2 + 128) * sizeof(cplx));   // b = 128
  static SmemLimit smem_limits[3];
  const int which = b <= 32 ? 0 : (b <= 64 ? 1 : 2);
  void (*const kernels[3])(const cplx*, int, const cplx*, cplx*, int, int, int, int, int, int) = {
      k_trsm_diag_block<1>, k_trsm_diag_block<2>, k_trsm_diag_block<4>};
  if (cudaError_t ea = smem_limits[which].raise((const void*)kernels[which], kMaxTdb); ea != cudaSuccess) return ea;
  // one column per warp and as few warps per SM as the m columns allow: a
  // solve is a chain of b FP64 steps, and warps that share a sub-partition
  // double it (m = 256, b = 64: 32 CTAs of 8 warps 48 and 79 us, lower and upper)
  int sms = 152;
  if (int dev = 0; cudaGetDevice(&dev) == cudaSuccess) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0) sms = v;
  }
  int warps = (m + sms - 1) / sms;
  if (warps > TRSM_DB_WARPS) warps = TRSM_DB_WARPS;
  kernels[which]<<<(m + warps - 1) / warps, 32 * TRSM_DB_WARPS, smem, st>>>(T, ldT, rdiag, Y, ldY, j0, b, m,
                                                                           lower ? 1 : 0, warps);
  return cudaGetLastError();
}

cudaError_t launch_wy_prep(const cplx* V, const cplx* tau, int n, int jb, int b, cplx* Vb, cplx* trd,
                           cudaStream_t st) {
  k_wy_prep<<<grid_for((size_t)(n - jb) * b), 256, 0, st>>>(V, tau, n, jb, b, Vb, trd);
  return cudaGetLastError();
}

cudaError_t launch_add(const cplx* A, const cplx* B, cplx* C, size_t count, cudaStream_t st) {
  k_add<<<grid_for(count), 256, 0, st>>>(A, B, C, count);
  return cudaGetLastError();
}

cudaError_t launch_iota(int* p, int n, cudaStream_t st) {
  k_iota<<<(n + 255) / 256, 256, 0, st>>>(p, n);
  return cudaGetLastError();
}

cudaError_t launch_split_scales(const double* Dl, const double* Dr, int n, double* s, cudaStream_t st) {
  k_split_scales<<<(n + 255) / 256, 256, 0, st>>>(Dl, Dr, n, s);
  return cudaGetLastError();
}

cudaError_t launch_lu_logdet(const cplx* udiag, const double* Dl, const double* Dr, int n, double* out,
                             cudaStream_t st) {
  k_lu_logdet<<<1, 256, 0, st>>>(udiag, Dl, Dr, n, out);
  return cudaGetLastError();
}

cudaError_t launch_trsm_right_upper(const cplx* T, const int* order, cplx* Y, int m, int n, cudaStream_t st) {
  size_t smem = (size_t)4 * n * sizeof(cplx);
  static SmemLimit smem_limit;
  if (cudaError_t ea = smem_limit.raise((const void*)k_trsm_right_upper, 200 * 1024); ea != cudaSuccess) return ea;
  k_trsm_right_upper<<<(m + 3) / 4, 128, smem, st>>>(T, order, Y, m, n);
  return cudaGetLastError();
}

cudaError_t launch_permute(const cplx* src, cplx* dst, int rows, int cols, const int* order, bool by_rows,
                           bool scatter, cudaStream_t st) {
  k_permute<<<grid_for((size_t)rows * cols), 256, 0, st>>>(src, dst, rows, cols, order, by_rows, scatter);
  return cudaGetLastError();
}

cudaError_t launch_add_diag(cplx* A, int n, const double* d, cudaStream_t st) {
  k_add_diag<<<(n + 255) / 256, 256, 0, st>>>(A, n, d);
  return cudaGetLastError();
}

cudaError_t launch_set_identity(cplx* A, int n, cudaStream_t st) {
  k_set_identity<<<grid_for((size_t)n * n), 256, 0, st>>>(A, n);
  return cudaGetLastError();
}

cudaError_t launch_scale(cplx* A, int rows, int cols, const double* rowscale, bool invert_rows,
                         const double* colscale, bool invert_cols, cudaStream_t st) {
  k_scale<<<grid_for((size_t)rows * cols), 256, 0, st>>>(A, rows, cols, rowscale, invert_rows, colscale,
                                                         invert_cols);
  return cudaGetLastError();
}

cudaError_t launch_conj_transpose(const cplx* A, cplx* B, int n, cudaStream_t st) {
  dim3 grid((n + 31) / 32, (n + 31) / 32);
  k_conj_transpose<<<grid, dim3(32, 8), 0, st>>>(A, B, n);
  return cudaGetLastError();
}

cudaError_t launch_sum_log(const double* x, int n, double* out, cudaStream_t st) {
  k_sum_log<<<1, 256, 0, st>>>(x, n, out);
  return cudaGetLastError();
}

__global__ void k_fill(double* d, int n, double v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = v;
}

cudaError_t launch_fill(double* d, int n, double v, cudaStream_t st) {
  k_fill<<<(n + 255) / 256, 256, 0, st>>>(d, n, v);
  return cudaGetLastError();
}

cudaError_t launch_max_absdiff(const cplx* A, const cplx* B, size_t count, double* out, cudaStream_t st, bool reset) {
  if (reset) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), st);
    if (e != cudaSuccess) return e;
  }
  k_max_absdiff<<<grid_for(count, 256, 1024), 256, 0, st>>>(A, B, count, out);
  return cudaGetLastError();
}
