// LU with partial pivoting (zgetrf / zgetf2 pivot rule: first row of maximal
// |Re| + |Im|) of the D-scale separated calculate_greens
// (src/stack.jl:338-369, src/linalg.jl:237-339).
#include <cooperative_groups.h>
#include "cluster.cuh"
#include "common.cuh"
#include "kernels.h"

namespace {

// Candidates compare on the bit patterns of the non-negative |Re| + |Im|, then
// on the row position.
__device__ __forceinline__ bool piv_better(double v, int r, double bv, int br) {
  const long long a = __double_as_longlong(v), b = __double_as_longlong(bv);   // v >= 0
  return a > b || (a == b && r < br);
}

__device__ __forceinline__ void warp_argmax(double& best, int& row) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int orow = __shfl_xor_sync(0xffffffffu, row, o);
    if (piv_better(ob, orow, best, row)) { best = ob; row = orow; }
  }
}


// a b with the multiply-adds spelled out: which product a compiler contracts
// depends on the context, and the forms of the LU have to agree bit for bit.
__device__ __forceinline__ cplx lu_mul(cplx a, cplx b) {
  return cmake(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}

constexpr int LU_THREADS = 256;
__device__ __forceinline__ void lu_bar() { asm volatile("bar.sync 1, 224;" ::: "memory"); }   // warps 1-7
constexpr int LU_LDP = LU_PB + 4;   // row stride of the panel in shared memory: 8 lanes on 2 rows x 4 columns miss no bank
constexpr int LU_MAXC = 16;

// A CTA's candidate in seven words, each with the step's tag in its high half, so
// that every word validates itself: the halves of |Re| + |Im|, position << 16 |
// row, and the halves of the candidate's real and imaginary part.
struct LuCand {
  unsigned long long w[8];
};
__device__ __forceinline__ double lu_join(unsigned hi, unsigned lo) { return __hiloint2double((int)hi, (int)lo); }

// Panel of b <= LU_PB columns [p0, p0 + b) over rows [p0, n) on one cluster of C
// CTAs, which hold the rows in contiguous chunks in shared memory.  Rows do not
// move: every CTA keeps the map between rows and their positions after the
// exchanges, and the rows go to their positions when the panel is written.
//
// Per column: everyone polls for all candidates and picks the same winner; one
// warp forms 1 / pivot while two others read the rest of the pivot row from its
// owner; then warp 0 updates the next column, finds this CTA's candidate in it
// and pushes it, beside the other warps' update of the remaining columns, whose
// end is pushed as well (the pivot row is read only after it).
//
// Bound: about 4500 cycles of latency per column (a remote store or load takes
// 1000, the reciprocal 1000-1500); the multiply-adds, 4 per entry on 16 SMs, fit
// beside them.  Panel of 64 columns, us: in turn -> overlapped n = 144 198 -> 178,
// n = 576 235 -> 190, n = 1024 229 -> 185.  The cooperative grids before paid a grid
// barrier and three round trips through L2 per column, 10000-15000 cycles.
//
// UNBLOCKED false: A in place, L below the diagonal (scaled multipliers, a -= l
// u), w.piv for the other columns.  true: the factors of zgetf2 as the trailing
// kernel continues it: the pivot row is scaled instead (a -= v (u / pivot)), A
// keeps v below the diagonal, L = v / pivot goes to Lb; w.src, w.perm, w.udiag and
// w.rdiag are written.
template <bool UNBLOCKED>
__global__ void __launch_bounds__(LU_THREADS) k_lu_panel(cplx* __restrict__ A, cplx* __restrict__ Lb, int n, int p0,
                                                        int b, LUPanel w) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), q = (int)cl.block_rank();
  const int R = n - p0, chunk = (R + C - 1) / C, r0 = q * chunk;
  const int nrw = max(0, min(R - r0, chunk));
  extern __shared__ double4_16a smem_lu[];
  cplx* prow = reinterpret_cast<cplx*>(smem_lu);             // (chunk, LU_LDP)
  int* pos = reinterpret_cast<int*>(prow + (size_t)chunk * LU_LDP);   // (R) row -> position
  int* rowat = pos + R;                                      // (R) position -> row
  __shared__ LuCand s_cand[2][LU_MAXC];
  __shared__ cplx urow[LU_PB], us[LU_PB], s_rinv[LU_PB], s_piv[LU_PB];   // us: urow / pivot
  __shared__ int s_win[2], s_pk[2], s_ready[LU_MAXC], s_late;   // s_ready: steps that CTA has finished
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int e = tid; e < nrw * b; e += LU_THREADS) {
    const int j = e / nrw, rr = e - j * nrw;
    prow[rr * LU_LDP + j] = ldcg_c(&A[(size_t)(p0 + j) * n + p0 + r0 + rr]);
  }
  for (int i = tid; i < R; i += LU_THREADS) { pos[i] = i; rowat[i] = i; }
  for (int e = tid; e < 2 * LU_MAXC * 8; e += LU_THREADS) s_cand[0][0].w[e] = 0ull;
  if (tid < LU_MAXC) s_ready[tid] = 0;
  if (tid == 0) s_late = 0;
  cl.sync();   // also: every CTA of the cluster runs before its shared memory is written remotely

  // warps 1-7: threads per row (chunk <= 128)
  const int tpr = max(1, (LU_THREADS - 32) / chunk);
  const int row = tid < 32 ? LU_THREADS : (tid - 32) / tpr, sub = (tid - 32) - row * tpr;
  const bool works = row < nrw && row * tpr + sub < LU_THREADS - 32;
  // warp 0: the candidate (or none) of this CTA for column kk, rows rr = lane, lane + 32, ...
  double best = 0.0;
  int pk = 0x7FFFFFFF;   // position << 16 | row; the positions of the candidates are distinct
  auto consider = [&](int kk, int rr, int ps, cplx x) {
    double a = fabs(x.x) + fabs(x.y);
    if (ps == kk && __double2hiint(a) < 0) a = 0.0;   // NaN: no candidate, but some row always is
    const int c = ps << 16 | (r0 + rr);
    if (piv_better(a, c, best, pk)) { best = a; pk = c; }
  };
  auto push = [&](int kk) {
    const int par = kk & 1;
    warp_argmax(best, pk);
    const bool any = pk != 0x7FFFFFFF;
    __syncwarp();
    const cplx x = any ? prow[((pk & 0xFFFF) - r0) * LU_LDP + kk] : cmake(0.0, 0.0);
    // lane c < 16 stores the first three words at CTA c, lane c + 16 the other four
    const int c = lane & 15;
    const unsigned long long tag = (unsigned long long)(kk + 1) << 32;
    if (c < C) {
      unsigned long long* o = cl.map_shared_rank(&s_cand[par][q].w[0], c);
      if (lane < 16) {
        st_cluster(o, tag | (unsigned)__double2hiint(best));
        st_cluster(o + 1, tag | (unsigned)__double2loint(best));
        st_cluster(o + 2, tag | (unsigned)pk);
      } else {
        st_cluster(o + 3, tag | (unsigned)__double2hiint(x.x));
        st_cluster(o + 4, tag | (unsigned)__double2loint(x.x));
        st_cluster(o + 5, tag | (unsigned)__double2hiint(x.y));
        st_cluster(o + 6, tag | (unsigned)__double2loint(x.y));
      }
    }
  };
  if (wid == 0) {
    for (int rr = lane; rr < nrw; rr += 32) consider(0, rr, r0 + rr, prow[rr * LU_LDP]);
    push(0);
  }
  bool ok = true, mine = false;
  cplx l = cmake(0.0, 0.0);
  for (int kk = 0; kk < b; ++kk) {
    const int par = kk & 1;
    cplx pvw = cmake(0.0, 0.0);   // warp 0: the pivot
    if (wid == 0) {
      // lane c polls CTA c's first three words, lane c + 16 the other four
      unsigned got[4] = {0u, 0u, 0u, 0u};
      bool here = false;
      for (int it = 0; it < kClusterPolls && !here; ++it) {
        bool all = true;
        if ((lane & 15) < C) {
          const int* m = reinterpret_cast<const int*>(&s_cand[par][lane & 15].w[lane < 16 ? 0 : 3]);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (u == 3 && lane < 16) break;
            got[u] = (unsigned)ld_poll(m + 2 * u);
            all = all && ld_poll(m + 2 * u + 1) == kk + 1;
          }
        }
        here = __all_sync(0xffffffffu, all);
        if (here) {   // the low halves are read again after the tags
          if ((lane & 15) < C) {
            const int* m = reinterpret_cast<const int*>(&s_cand[par][lane & 15].w[lane < 16 ? 0 : 3]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (u < 3 || lane >= 16) got[u] = (unsigned)ld_poll(m + 2 * u);
          }
        }
      }
      __syncwarp();
      best = 0.0;
      pk = 0x7FFFFFFF;
      int win = 0;
      if (lane < C) {
        best = lu_join(got[0], got[1]);
        pk = (int)got[2];
        win = lane;
      }
#pragma unroll
      for (int o = LU_MAXC / 2; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int op = __shfl_xor_sync(0xffffffffu, pk, o), ow = __shfl_xor_sync(0xffffffffu, win, o);
        if (piv_better(ob, op, best, pk)) { best = ob; pk = op; win = ow; }
      }
      win = __shfl_sync(0xffffffffu, win, 0);
      pvw = cmake(__shfl_sync(0xffffffffu, lu_join(got[0], got[1]), win + 16),
                  __shfl_sync(0xffffffffu, lu_join(got[2], got[3]), win + 16));
      if (lane == 0) {
        s_win[par] = here ? win : -1;
        s_pk[par] = pk;
      }
    }
    __syncthreads();
    const int win = s_win[par], pkw = s_pk[par];
    if (win < 0) { ok = false; break; }
    // column kk - 1 is read no more: its multipliers take their place
    if (!UNBLOCKED && mine && sub == 0) prow[(size_t)row * LU_LDP + kk - 1] = l;
    const int ps = pkw >> 16, o = pkw & 0xFFFF;
    if (wid == 0) {
      const cplx pv = pvw;
      bool zero = pv.x == 0.0 && pv.y == 0.0;
      cplx ri;
      if (UNBLOCKED) {
        ri = zero ? cmake(0.0, 0.0) : cdiv(cmake(1.0, 0.0), pv);
      } else {
        // 1 / pivot = conj(pv) / |pv|^2 (the D-scale separated matrix has no large scales)
        const double d2 = pv.x * pv.x + pv.y * pv.y;
        zero = d2 == 0.0;   // also a pivot below 1e-162, which has no reciprocal here
        const double rd = zero ? 0.0 : 1.0 / d2;
        ri = cmake(pv.x * rd, -pv.y * rd);
      }
      if (lane == 0) {
        s_rinv[kk] = ri;
        s_piv[kk] = pv;
        if (zero && q == 0) atomicOr(w.err, DQMC_KERR_SINGULAR);
        if (!UNBLOCKED && q == 0) w.piv[p0 + kk] = p0 + ps;
      }
    } else if (wid <= 2) {
      // the pivot row, once its CTA has finished the step before
      bool here = false;
      for (int it = 0; it < kClusterPolls && !here; ++it) here = ld_poll(&s_ready[win]) >= kk;
      fence_acquire_shared();
      __syncwarp();
      if (!here && lane == 0) s_late = 1;
      const int j = tid - 32;
      if (j > kk && j < b) urow[j] = cl.map_shared_rank(prow + (size_t)(o - win * chunk) * LU_LDP, win)[j];
    } else if (wid == 3 && lane == 0) {
      const int o2 = rowat[kk];
      pos[o] = kk;
      pos[o2] = o2 == o ? kk : ps;
      rowat[ps] = o2;
      rowat[kk] = o;
    }
    __syncthreads();
    if (wid == 0) {
      // column kk + 1 ahead of the others: its candidate is on its way while they work
      best = 0.0;
      pk = 0x7FFFFFFF;
      if (kk + 1 < b) {
        const cplx ri = s_rinv[kk];
        const cplx u = UNBLOCKED ? lu_mul(urow[kk + 1], ri) : urow[kk + 1];
        for (int rr = lane; rr < nrw; rr += 32) {
          const int pr_pos = pos[r0 + rr];
          if (pr_pos <= kk) continue;
          cplx* pr = prow + (size_t)rr * LU_LDP;
          const cplx lw = UNBLOCKED ? pr[kk] : lu_mul(pr[kk], ri), x0 = pr[kk + 1];
          const cplx x = cmake(fma(-lw.x, u.x, fma(lw.y, u.y, x0.x)), fma(-lw.x, u.y, fma(-lw.y, u.x, x0.y)));
          pr[kk + 1] = x;
          consider(kk + 1, rr, pr_pos, x);
        }
        push(kk + 1);
      }
    } else {
      if (UNBLOCKED) {
        const int j = tid - 32;
        if (j > kk && j < b) us[j] = lu_mul(urow[j], s_rinv[kk]);
        lu_bar();
      }
      const cplx* uu = UNBLOCKED ? us : urow;
      mine = works && pos[r0 + row] > kk;
      if (mine) {
        cplx* pr = prow + (size_t)row * LU_LDP;
        l = UNBLOCKED ? pr[kk] : lu_mul(pr[kk], s_rinv[kk]);
        for (int j = kk + 2 + sub; j < b; j += tpr) {
          const cplx u = uu[j], x = pr[j];
          pr[j] = cmake(fma(-l.x, u.x, fma(l.y, u.y, x.x)), fma(-l.x, u.y, fma(-l.y, u.x, x.y)));
        }
      }
      lu_bar();
      if (wid == 1) {
        fence_release_shared();   // this CTA's rows
        if (lane < C) st_cluster(cl.map_shared_rank(&s_ready[q], lane), kk + 1);
      }
    }
  }
  __syncthreads();
  if (ok && !UNBLOCKED && mine && sub == 0) prow[(size_t)row * LU_LDP + b - 1] = l;
  ok = ok && s_late == 0;
  if (!ok && tid == 0) atomicOr(w.err, DQMC_KERR_BARRIER_TIMEOUT);
  __syncthreads();
  if (ok) {
    for (int e = tid; e < nrw * b; e += LU_THREADS) {
      const int j = e / nrw, rr = e - j * nrw, ps = pos[r0 + rr];
      const cplx x = prow[rr * LU_LDP + j];
      A[(size_t)(p0 + j) * n + p0 + ps] = x;
      if (UNBLOCKED && ps > j) Lb[(size_t)(p0 + j) * n + p0 + ps] = lu_mul(x, s_rinv[j]);
    }
    if (UNBLOCKED && q == 0) {
      __syncthreads();   // pos has been read by all warps
      if (tid < b) {
        w.udiag[p0 + tid] = s_piv[tid];
        w.rdiag[p0 + tid] = s_rinv[tid];
      }
      for (int i = tid; i < R; i += LU_THREADS) {
        w.src[i] = rowat[i];
        pos[i] = p0 == 0 ? rowat[i] : w.perm[p0 + rowat[i]];
      }
      __syncthreads();
      for (int i = tid; i < R; i += LU_THREADS) w.perm[p0 + i] = pos[i];
    }
  }
  cl.sync();   // no shared memory is read remotely any more
}

// The unblocked LU continued over the columns right of a panel (UNBLOCKED
// above), CW columns per CTA: the panel's row order, the top b rows solved
// column step by column step, and the rows below updated, every entry by the
// same multiply-adds in the same order as a column-at-a-time elimination.  The
// last p0 blocks bring the multiplier columns left of the panel into the
// panel's row order.  Bound: FP64 issue, 4 multiply-adds per entry and step.
template <int CW>
__global__ void __launch_bounds__(LU_THREADS) k_lu_trail(cplx* __restrict__ A, cplx* __restrict__ Lb, int n, int p0,
                                                        int b, const int* __restrict__ src,
                                                        const cplx* __restrict__ rdiag) {
  extern __shared__ double4_16a smem_lt[];
  cplx* X = reinterpret_cast<cplx*>(smem_lt);   // (CW, R)
  const int R = n - p0, tid = threadIdx.x;
  const int groups = (n - p0 - b + CW - 1) / CW;
  if ((int)blockIdx.x >= groups) {
    cplx* col = Lb + (size_t)(blockIdx.x - groups) * n + p0;
    for (int i = tid; i < R; i += LU_THREADS) X[i] = ldcg_c(&col[src[i]]);
    __syncthreads();
    for (int i = tid; i < R; i += LU_THREADS) col[i] = X[i];
    return;
  }
  cplx* V = X + (size_t)CW * R;                 // (b, b + 1): V[k][i] = v of step k, row i < b
  cplx* cs = V + (size_t)LU_PB * (LU_PB + 1);   // (b, CW): u / pivot
  const int c0 = p0 + b + blockIdx.x * CW, nc = min(CW, n - c0);
  for (int e = tid; e < CW * R; e += LU_THREADS) {
    const int c = e / R, i = e - c * R;
    X[e] = c < nc ? ldcg_c(&A[(size_t)(c0 + c) * n + p0 + src[i]]) : cmake(0.0, 0.0);
  }
  for (int e = tid; e < b * b; e += LU_THREADS) {
    const int k = e / b, i = e - k * b;
    if (i > k) V[k * (LU_PB + 1) + i] = ldcg_c(&A[(size_t)(p0 + k) * n + p0 + i]);
  }
  __syncthreads();
  // top rows: thread (i, c) holds row i of column c
  const int i1 = tid / CW, c1 = tid - i1 * CW;
  constexpr int ROWS = LU_THREADS / CW;         // rows per pass (>= LU_PB)
  static_assert(ROWS >= LU_PB, "one pass over the top rows");
  cplx x = i1 < b ? X[c1 * R + i1] : cmake(0.0, 0.0);
  for (int k = 0; k < b; ++k) {
    if (i1 == k) {
      X[c1 * R + k] = x;
      cs[k * CW + c1] = lu_mul(x, __ldg(&rdiag[p0 + k]));
    }
    __syncthreads();
    if (i1 > k && i1 < b) {
      const cplx vr = V[k * (LU_PB + 1) + i1], c = cs[k * CW + c1];
      x = cmake(fma(-vr.x, c.x, fma(vr.y, c.y, x.x)), fma(-vr.x, c.y, fma(-vr.y, c.x, x.y)));
    }
  }
  __syncthreads();
  // rows below
  for (int i = b + tid; i < R; i += LU_THREADS) {
    cplx y[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) y[c] = X[c * R + i];
    const cplx* v = A + (size_t)p0 * n + p0 + i;
#pragma unroll 4
    for (int k = 0; k < b; ++k) {
      const cplx vr = ldcg_c(&v[(size_t)k * n]);
#pragma unroll
      for (int c = 0; c < CW; ++c) {
        const cplx u = cs[k * CW + c];
        y[c] = cmake(fma(-vr.x, u.x, fma(vr.y, u.y, y[c].x)), fma(-vr.x, u.y, fma(-vr.y, u.x, y[c].y)));
      }
    }
#pragma unroll
    for (int c = 0; c < CW; ++c) X[c * R + i] = y[c];
  }
  __syncthreads();
  for (int e = tid; e < nc * R; e += LU_THREADS) {
    const int c = e / R, i = e - c * R;
    A[(size_t)(c0 + c) * n + p0 + i] = X[e];
  }
}

// Row exchanges of one panel applied to the columns outside it, and to the
// running permutation: the b exchanges (k, piv[k]) touch at most 2b rows,
// whose net permutation warp 0 works out (panel rows indexed directly, rows
// below the panel found by a ballot over the ones met so far); every column
// is then gathered over those rows.
__global__ void k_lu_apply_swaps(cplx* __restrict__ A, int n, int p0, int b, const int* __restrict__ piv,
                                 int* __restrict__ perm) {
  __shared__ int rowof[2 * LU_PB], src[2 * LU_PB], spiv[LU_PB];
  __shared__ int s_cnt;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    for (int s2 = lane; s2 < b; s2 += 32) {
      rowof[s2] = p0 + s2;
      src[s2] = p0 + s2;
      spiv[s2] = piv[p0 + s2];
    }
    __syncwarp();
    int cnt = b;
    for (int kk = 0; kk < b; ++kk) {
      const int k = p0 + kk, pr = spiv[kk];
      if (pr == k) continue;   // warp-uniform
      int sp = -1;
      if (pr < p0 + b) {
        sp = pr - p0;
      } else {
        for (int base = b; base < cnt && sp < 0; base += 32) {
          const int s2 = base + lane;
          const unsigned hit = __ballot_sync(0xffffffffu, s2 < cnt && rowof[s2] == pr);
          if (hit) sp = base + __ffs(hit) - 1;
        }
        if (sp < 0) {
          sp = cnt++;
          if (lane == 0) { rowof[sp] = pr; src[sp] = pr; }
        }
      }
      __syncwarp();
      if (lane == 0) { const int t = src[kk]; src[kk] = src[sp]; src[sp] = t; }
      __syncwarp();
    }
    if (lane == 0) s_cnt = cnt;
  }
  __syncthreads();
  const int cnt = s_cnt;
  // permutation (block 0): perm[rowof[s]] <- old perm[src[s]]
  if (blockIdx.x == 0) {
    __shared__ int pv[2 * LU_PB];
    for (int s2 = threadIdx.x; s2 < cnt; s2 += blockDim.x) pv[s2] = perm[src[s2]];
    __syncthreads();
    for (int s2 = threadIdx.x; s2 < cnt; s2 += blockDim.x) perm[rowof[s2]] = pv[s2];
  }
  // columns outside the panel, one warp per column
  const int lane = threadIdx.x & 31;
  const int nw = blockDim.x >> 5;
  for (int c = blockIdx.x * nw + (threadIdx.x >> 5); c < n; c += gridDim.x * nw) {
    if (c >= p0 && c < p0 + b) continue;
    cplx* col = A + (size_t)c * n;
    cplx v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int s2 = lane + 32 * q;
      if (s2 < cnt) v[q] = ldcg_c(&col[src[s2]]);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int s2 = lane + 32 * q;
      if (s2 < cnt) col[rowof[s2]] = v[q];
    }
  }
}

// udiag = diag(U) of the in-place LU, rdiag = 1 / udiag
__global__ void k_lu_diag(const cplx* __restrict__ A, int n, cplx* __restrict__ udiag, cplx* __restrict__ rdiag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const cplx d = A[(size_t)i * n + i];
    udiag[i] = d;
    rdiag[i] = (d.x == 0.0 && d.y == 0.0) ? cmake(0.0, 0.0) : cdiv(cmake(1.0, 0.0), d);
  }
}

}  // namespace

// One cluster of 16 CTAs, else 8 (the size is asked of the device once); cs > 0
// asks for at most that many.
template <bool UNBLOCKED>
static cudaError_t launch_panel(cplx* A, cplx* Lb, int n, int p0, int b, const LUPanel& w, int cs, cudaStream_t st) {
  if (b < 1 || b > LU_PB || n - p0 > 1024 || n - p0 < b) return cudaErrorInvalidValue;
  const void* fn = (const void*)k_lu_panel<UNBLOCKED>;
  auto smem_of = [](int R, int c) {
    const int chunk = (R + c - 1) / c;
    return (size_t)chunk * LU_LDP * sizeof(cplx) + (size_t)2 * R * sizeof(int);
  };
  auto config = [&](cudaLaunchAttribute* attr, int c, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(LU_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
  };
  static std::mutex mu;
  static int cached[64] = {};
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] == 0) {
      if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1); e != cudaSuccess)
        return e;
      if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_of(1024, 8));
          e != cudaSuccess)
        return e;
      for (int c = LU_MAXC; c >= 8 && cached[dev] == 0; c /= 2) {
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = config(attr, c, smem_of(1024, c));
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
          cudaGetLastError();
          clusters = 0;
        }
        if (clusters >= 1) cached[dev] = c;
      }
      if (cached[dev] == 0) return cudaErrorNotSupported;
    }
  }
  int c = cached[dev];
  if (cs > 0 && cs < c) c = 8;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = config(attr, c, smem_of(n - p0, c));
  return cudaLaunchKernelEx(&cfg, k_lu_panel<UNBLOCKED>, A, Lb, n, p0, b, w);
}

cudaError_t launch_lu_panel(cplx* A, int n, int p0, int b, const LUPanel& w, int max_cluster, cudaStream_t st) {
  return launch_panel<false>(A, nullptr, n, p0, b, w, max_cluster, st);
}

cudaError_t launch_lu_unblocked_panel(cplx* A, cplx* Lb, int n, int p0, int b, const LUPanel& w, int max_cluster,
                                      cudaStream_t st) {
  return launch_panel<true>(A, Lb, n, p0, b, w, max_cluster, st);
}

cudaError_t launch_lu_trail(cplx* A, cplx* Lb, int n, int p0, int b, const LUPanel& w, cudaStream_t st) {
  const int rest = n - p0 - b;
  // columns per CTA: as few as keep the grid near one CTA per SM
  const int cw = rest <= 160 ? 1 : (rest <= 320 ? 2 : 4);
  const int groups = (rest + cw - 1) / cw, grid = groups + p0;
  if (grid < 1) return cudaSuccess;
  const size_t smem = ((size_t)cw * (n - p0) + LU_PB * (LU_PB + 1) + LU_PB * cw) * sizeof(cplx);
  static SmemLimit limits[3];
  const int which = cw == 1 ? 0 : (cw == 2 ? 1 : 2);
  void (*const fns[3])(cplx*, cplx*, int, int, int, const int*, const cplx*) = {k_lu_trail<1>, k_lu_trail<2>,
                                                                               k_lu_trail<4>};
  if (cudaError_t e = limits[which].raise((const void*)fns[which], (int)smem); e != cudaSuccess) return e;
  fns[which]<<<grid, LU_THREADS, smem, st>>>(A, Lb, n, p0, b, w.src, w.rdiag);
  return cudaGetLastError();
}

cudaError_t launch_lu_apply_swaps(cplx* A, int n, int p0, int b, const int* piv, int* perm, cudaStream_t st) {
  k_lu_apply_swaps<<<(n + 7) / 8, 256, 0, st>>>(A, n, p0, b, piv, perm);
  return cudaGetLastError();
}

cudaError_t launch_lu_diag(const cplx* A, int n, cplx* udiag, cplx* rdiag, cudaStream_t st) {
  k_lu_diag<<<(n + 255) / 256, 256, 0, st>>>(A, n, udiag, rdiag);
  return cudaGetLastError();
}

