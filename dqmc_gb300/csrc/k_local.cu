// Local Metropolis updates of one time slice: windows of sites with their
// factors and flush (the handle's updates, see "windows of sites" below), and
// immediate rank-4 updates (the allocation-free entry point).
//
// Reference: src/local_updates.jl:1-95 (local_updates, calc_detratio,
// update_greens!), src/action.jl:57-100 (calc_boson_action_diff),
// src/interactions.jl:102-141 (interaction_matrix_exp_op!).
//
// Immediate form: one cooperative (co-resident) launch visits all N sites of the
// slice in order.  Structure:
//   * prologue: every CTA builds, for all sites in parallel, the 4x4 block
//     Delta_i = e^{+dtau V(phi_i)} e^{-dtau V(phi_i + delta_i)} - I into shared
//     memory (the old field of a site cannot change before its own visit);
//   * per site, warp 0 of every CTA evaluates the ratio redundantly and
//     identically from the same 16 entries of G: lanes build
//     M = I + Delta (I - G_ii) entry-wise, 24 lanes form the permutation
//     expansion of det M, and on acceptance 16 lanes form M^-1 = adj(M)/det;
//     all CTAs therefore take the same decision without communicating;
//   * on acceptance the rank-4 update G += A B, A = (G[:,c] - I[:,c]) M^-1
//     (n x 4), B = Delta G[r,:] (4 x n), runs over the whole grid in two phases
//     separated by grid barriers: phase 1 forms A and B from the unmodified G,
//     phase 2 applies them with warp tiles of 128 rows x 4 columns (A held in
//     registers, B broadcast).  Rejected sites cost no barrier.
//
// Proposal streams use fixed slots: delta[:, i] and unif[i] belong to site
// i of this call; unif[i] decides only when p_acc <= 1, exactly as
// `p_acc > 1.0 || rand() < p_acc`.
#include <algorithm>
#include <cooperative_groups.h>
#include "cluster.cuh"
#include "common.cuh"
#include "kernels.h"
#include "oz_slice.cuh"

namespace {

// The 24 permutations of (0,1,2,3) and their signs, for det M.
__constant__ unsigned char c_perm[24][4] = {
    {0, 1, 2, 3}, {0, 1, 3, 2}, {0, 2, 1, 3}, {0, 2, 3, 1}, {0, 3, 1, 2}, {0, 3, 2, 1},
    {1, 0, 2, 3}, {1, 0, 3, 2}, {1, 2, 0, 3}, {1, 2, 3, 0}, {1, 3, 0, 2}, {1, 3, 2, 0},
    {2, 0, 1, 3}, {2, 0, 3, 1}, {2, 1, 0, 3}, {2, 1, 3, 0}, {2, 3, 0, 1}, {2, 3, 1, 0},
    {3, 0, 1, 2}, {3, 0, 2, 1}, {3, 1, 0, 2}, {3, 1, 2, 0}, {3, 2, 0, 1}, {3, 2, 1, 0}};
__constant__ signed char c_psign[24] = {1, -1, -1, 1, 1, -1, -1, 1, 1, -1, -1, 1,
                                         1, -1, -1, 1, 1, -1, -1, 1, 1, -1, -1, 1};

// Interaction block parameters of exp(-power*dtau*V(op)) for one site
// (src/interactions.jl:102-141): C, S, R with S, R scaled by `power`.
__device__ __forceinline__ void ev_params(const ModelConst& mc, const double op[3], double power, double& C,
                                          cplx& S, double& R, double& shn) {
  double nrm = sqrt(op[0] * op[0] + op[1] * op[1] + op[2] * op[2]);
  double a = mc.lambda * mc.dtau * nrm;
  shn = sinh(a) / nrm;
  C = cosh(a);
  double sh = power * shn;
  S = cmake(-op[0] * sh, op[1] * sh);
  R = -op[2] * sh;
}

// Entry (r, c) of the block [[C,S,0,R],[S*,C,-R,0],[0,-R,C,S*],[R,0,S,C]].
__device__ __forceinline__ cplx ev_entry(int r, int c, double C, cplx S, double R) {
  const int code = r * 4 + c;
  switch (code) {
    case 0: case 5: case 10: case 15: return cmake(C, 0.0);
    case 1: case 14: return S;
    case 4: case 11: return cconj(S);
    case 3: case 12: return cmake(R, 0.0);
    case 6: case 9: return cmake(-R, 0.0);
    default: return cmake(0.0, 0.0);
  }
}

__device__ __forceinline__ cplx shfl_c(cplx v, int src) {
  return cmake(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

struct SiteDecision {
  int accepted;
  cplx minv[4][4];
};

constexpr int LU_THREADS = 256;

// Shared-memory layout of both local-update kernels.
struct LocalSmem {
  cplx* delta_all;   // (N, 16): Delta_i row-major
  EvEntry* evnew;    // (N): interaction entries of the proposed field
  double* phis;      // (3, N): this CTA's copy of phi[:, :, l]
};

__device__ LocalSmem local_smem(void* base, int N) {
  LocalSmem s;
  s.delta_all = reinterpret_cast<cplx*>(base);
  s.evnew = reinterpret_cast<EvEntry*>(s.delta_all + 16 * N);
  s.phis = reinterpret_cast<double*>(s.evnew + N);
  return s;
}

// Field copy of slice l and Delta_i = e^{+dtau V(phi_i)} e^{-dtau V(phi_i + delta_i)} - I
// for sites >= first (the old field of a site cannot change before its visit).
__device__ void local_prologue(const LocalUpdateArgs& a, const LocalSmem& sm, int first) {
  const ModelConst& mc = a.mc;
  const int N = mc.N, l = a.slice0;
  for (int k = threadIdx.x; k < 3 * N; k += blockDim.x) sm.phis[k] = a.phi[(size_t)3 * N * l + k];
  for (int i = first + threadIdx.x; i < N; i += blockDim.x) {
    const double* po = &a.phi[((size_t)N * l + i) * 3];
    double old[3] = {po[0], po[1], po[2]};
    double nw[3] = {old[0] + a.delta[3 * i], old[1] + a.delta[3 * i + 1], old[2] + a.delta[3 * i + 2]};
    double C1, R1, s1, C2, R2, s2;
    cplx S1, S2;
    ev_params(mc, old, -1.0, C1, S1, R1, s1);
    ev_params(mc, nw, 1.0, C2, S2, R2, s2);
    EvEntry e;
    e.C = C2; e.Sr = -nw[0] * s2; e.Si = nw[1] * s2; e.R = -nw[2] * s2;
    sm.evnew[i] = e;
    for (int r = 0; r < 4; ++r)
      for (int c = 0; c < 4; ++c) {
        cplx s = cmake(0.0, 0.0);
        for (int k = 0; k < 4; ++k) s = cfma(ev_entry(r, k, C1, S1, R1), ev_entry(k, c, C2, S2, R2), s);
        if (r == c) s.x -= 1.0;
        sm.delta_all[16 * i + 4 * r + c] = s;
      }
  }
}

// Metropolis decision for site i, executed by warp 0 of every CTA.  g is
// G_cur[i + rN, i + cN] in lane 4r + c (lanes < 16).  Writes dec (accepted
// flag, M^-1), the CTA's field copy, and (CTA 0) the outputs, the field,
// the interaction table, the action and the accepted count.
__device__ void local_decide(const LocalUpdateArgs& a, const LocalSmem& sm, int i, cplx g, SiteDecision& dec) {
  const ModelConst& mc = a.mc;
  const int N = mc.N, M = mc.M, L = mc.L, l = a.slice0;
  const int lane = threadIdx.x & 31;
  const int lt_later = (l + 1) % M, lt_earlier = (l - 1 + M) % M;
  double* phis = sm.phis;
  // ---- boson action difference (src/action.jl:57-100), lane 0 ----
  double dS = 0.0;
  if (lane == 0) {
    double old[3] = {phis[3 * i], phis[3 * i + 1], phis[3 * i + 2]};
    double nw[3];
    for (int c = 0; c < 3; ++c) nw[c] = old[c] + a.delta[3 * i + c];
    double diff[3] = {nw[0] - old[0], nw[1] - old[1], nw[2] - old[2]};
    double old_sq = old[0] * old[0] + old[1] * old[1] + old[2] * old[2];
    double new_sq = nw[0] * nw[0] + nw[1] * nw[1] + nw[2] * nw[2];
    double sq_diff = new_sq - old_sq;
    double pow4_diff = new_sq * new_sq - old_sq * old_sq;
    const double* pe = (lt_earlier == l) ? &phis[3 * i] : &a.phi[((size_t)N * lt_earlier + i) * 3];
    const double* pl = (lt_later == l) ? &phis[3 * i] : &a.phi[((size_t)N * lt_later + i) * 3];
    int y = i % L, x = i / L;
    int nbs[4] = {(y + 1) % L + L * x, y + L * ((x + 1) % L), (y - 1 + L) % L + L * x, y + L * ((x - 1 + L) % L)};
    double tdot = 0.0, sdot = 0.0;
    for (int c = 0; c < 3; ++c) {
      double ot = pl[c] + pe[c];
      double os = 0.0;
      for (int q = 0; q < 4; ++q) os = os + phis[3 * nbs[q] + c];
      tdot += ot * diff[c];
      sdot += os * diff[c];
    }
    dS += 1.0 / (mc.dtau * mc.c * mc.c) * (sq_diff - tdot);
    dS += 0.5 * mc.dtau * (4 * sq_diff - 2.0 * sdot);
    dS += mc.dtau * (0.5 * mc.r * sq_diff + 0.25 * mc.u * pow4_diff);
  }
  dS = __shfl_sync(0xffffffffu, dS, 0);
  // ---- M = I + Delta (I - G_ii), lane 4r+c holds M[r][c] (src/local_updates.jl:49-55) ----
  const int r = (lane >> 2) & 3, c = lane & 3;
  if (lane >= 16) g = cmake(0.0, 0.0);
  cplx mt = cmake((r == c ? 1.0 : 0.0) - g.x, -g.y);   // (I - G_ii)[r][c]
  cplx m = cmake(r == c ? 1.0 : 0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    cplx mtk = shfl_c(mt, 4 * k + c);                  // (I - G_ii)[k][c]
    m = cfma(sm.delta_all[16 * i + 4 * r + k], mtk, m);
  }
  // ---- det M by the permutation expansion (24 lanes) ----
  cplx term = cmake(0.0, 0.0);
  {
    const int j = lane < 24 ? lane : 0;
    cplx p = cmake(1.0, 0.0);
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) p = cmul(p, shfl_c(m, 4 * rr + c_perm[j][rr]));
    if (lane < 24) term = cscale(p, (double)c_psign[j]);
  }
  cplx det = term;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) det = cadd(det, shfl_c(det, lane ^ o));
  // lanes associate the sum differently; lane 0's value (the same in every
  // CTA) is the one every lane uses, so all decisions agree bit for bit
  det = shfl_c(det, 0);
  const double exp_dS = exp(-dS);
  const double pacc = exp_dS * det.x;
  const double u = a.unif[i];
  int acc = (pacc > 1.0 || u < pacc) ? 1 : 0;
  const bool bad = !isfinite(det.x) || !isfinite(det.y) || (det.x == 0.0 && det.y == 0.0);
  if (bad) acc = 0;
  // ---- M^-1 = adj(M) / det (lane 4r+c: entry [r][c] = cofactor C[c][r] / det) ----
  if (acc) {
    int rows[3], cols[3];
    for (int t = 0, q = 0; t < 4; ++t) if (t != c) rows[q++] = t;
    for (int t = 0, q = 0; t < 4; ++t) if (t != r) cols[q++] = t;
    cplx e[3][3];
#pragma unroll
    for (int u3 = 0; u3 < 3; ++u3)
#pragma unroll
      for (int v3 = 0; v3 < 3; ++v3) e[u3][v3] = shfl_c(m, (4 * rows[u3] + cols[v3]) & 31);
    cplx d3 = csub(cmul(e[0][0], csub(cmul(e[1][1], e[2][2]), cmul(e[1][2], e[2][1]))),
                   cmul(e[0][1], csub(cmul(e[1][0], e[2][2]), cmul(e[1][2], e[2][0]))));
    d3 = cadd(d3, cmul(e[0][2], csub(cmul(e[1][0], e[2][1]), cmul(e[1][1], e[2][0]))));
    if ((r + c) & 1) d3 = cmake(-d3.x, -d3.y);
    if (lane < 16) dec.minv[r][c] = cdiv(d3, det);
  }
  if (lane == 0) {
    dec.accepted = acc;
    if (acc) {
      for (int q = 0; q < 3; ++q) phis[3 * i + q] += a.delta[3 * i + q];
    }
    if (blockIdx.x == 0) {
      if (bad) atomicOr(a.err, DQMC_KERR_NONFINITE);
      if (a.acc_out) a.acc_out[i] = (uint8_t)acc;
      if (a.det_out) a.det_out[i] = det;
      if (a.pacc_out) a.pacc_out[i] = pacc;
      if (acc) {
        double* pg = &a.phi[((size_t)N * l + i) * 3];
        pg[0] = phis[3 * i]; pg[1] = phis[3 * i + 1]; pg[2] = phis[3 * i + 2];
        if (a.evtab) reinterpret_cast<EvEntry*>(a.evtab)[(size_t)N * l + i] = sm.evnew[i];
        *a.action += -log(exp_dS);
        *a.n_acc += 1;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// immediate rank-4 updates
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(LU_THREADS, 2) k_local_updates(LocalUpdateArgs a) {
  unsigned bar_epoch = 0;
  GridBarrierExit bar_exit(a.bar);
  const ModelConst& mc = a.mc;
  const int N = mc.N, n = mc.n;
  extern __shared__ double4_16a smem_local[];
  const LocalSmem sm = local_smem(smem_local, N);
  __shared__ SiteDecision dec;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  local_prologue(a, sm, 0);
  __syncthreads();
  const int gwarp = blockIdx.x * (LU_THREADS / 32) + wid;
  const int nwarps = gridDim.x * (LU_THREADS / 32);

  for (int i = 0; i < N; ++i) {
    if (wid == 0) {
      const int r = (lane >> 2) & 3, c = lane & 3;
      cplx g = cmake(0.0, 0.0);
      if (lane < 16) g = ldcg_c(&a.G[(size_t)(i + c * N) * n + i + r * N]);
      local_decide(a, sm, i, g, dec);
    }
    __syncthreads();
    const int accepted = dec.accepted;
    if (!accepted) {
      __syncthreads();   // every thread has read the decision before warp 0 overwrites it
      continue;
    }
    // ---- phase 1: A = (G[:, cols] - I[:, cols]) M^-1, B = Delta G[rows, :] ----
    const cplx* Dl = &sm.delta_all[16 * i];
    for (int t = blockIdx.x * LU_THREADS + threadIdx.x; t < 2 * n; t += gridDim.x * LU_THREADS) {
      if (t < n) {
        const int row = t;
        cplx g[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          g[k] = ldcg_c(&a.G[(size_t)(i + k * N) * n + row]);
          if (row == i + k * N) g[k].x -= 1.0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          cplx s = cmake(0, 0);
#pragma unroll
          for (int k = 0; k < 4; ++k) s = cfma(g[k], dec.minv[k][c], s);
          a.Acol[(size_t)c * n + row] = s;
        }
      } else {
        const int col = t - n;
        cplx g[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) g[k] = ldcg_c(&a.G[(size_t)col * n + i + k * N]);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          cplx s = cmake(0, 0);
#pragma unroll
          for (int k = 0; k < 4; ++k) s = cfma(Dl[4 * r + k], g[k], s);
          a.Brow[(size_t)r * n + col] = s;
        }
      }
    }
    if (!grid_barrier(a.bar, a.err, bar_epoch)) return;
    // ---- phase 2: G += A B over warp tiles of 128 rows x 4 columns ----
    const int tiles_r = (n + 127) / 128, tiles_c = (n + 3) / 4;
    for (int tile = gwarp; tile < tiles_r * tiles_c; tile += nwarps) {
      const int tr = tile % tiles_r, tc = tile / tiles_r;
      const int r0 = tr * 128 + lane, c0 = tc * 4;
      cplx Av[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int row = r0 + 32 * q;
#pragma unroll
        for (int k = 0; k < 4; ++k) Av[q][k] = row < n ? ldcg_c(&a.Acol[(size_t)k * n + row]) : cmake(0, 0);
      }
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        const int col = c0 + cc;
        if (col >= n) break;
        cplx Bv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) Bv[k] = ldcg_c(&a.Brow[(size_t)k * n + col]);
        cplx* gcol = a.G + (size_t)col * n;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int row = r0 + 32 * q;
          if (row < n) {
            cplx v = ldcg_c(&gcol[row]);
#pragma unroll
            for (int k = 0; k < 4; ++k) v = cfma(Av[q][k], Bv[k], v);
            gcol[row] = v;
          }
        }
      }
    }
    if (!grid_barrier(a.bar, a.err, bar_epoch)) return;
  }
}

// ---------------------------------------------------------------------------
// delayed updates: windows of sites decided on one thread-block cluster
// ---------------------------------------------------------------------------
// A round takes the next W sites of the slice (a window).  The Metropolis
// decisions of its sites need G only on the window's own 4W rows and columns,
// so one cluster keeps that block in shared memory and decides the window
// there (k_local_window); the whole chip then forms the rank-4p factors of the
// p accepted sites (k_local_factors) and applies them as one product (flush).
// Per-site constants of slice l: one warp per site.  Lanes of even parity
// evaluate the old-field block (power -1), odd lanes the proposed one.
__global__ void __launch_bounds__(128) k_local_prepare(LocalUpdateArgs a, SitePrep* __restrict__ prep, int* state,
                                                       int* wflag) {
  const ModelConst& mc = a.mc;
  const int N = mc.N, M = mc.M, l = a.slice0;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
  // delayed rounds of this slice start from site 0 with nothing pending
  if (blockIdx.x == 0 && threadIdx.x == 0) { state[0] = 0; state[1] = 0; state[2] = 0; }
  // flags carry the window's first site; the last two are the arrivals, which a
  // window that timed out leaves behind (no window is in flight here)
  if (blockIdx.x == 0 && threadIdx.x < WIN_MAX + 3) wflag[threadIdx.x] = 0;
  if (i >= N) return;
  const double* po = &a.phi[((size_t)N * l + i) * 3];
  const double old[3] = {po[0], po[1], po[2]};
  const double nw[3] = {old[0] + a.delta[3 * i], old[1] + a.delta[3 * i + 1], old[2] + a.delta[3 * i + 2]};
  const bool odd = lane & 1;
  double C, R, shn;
  cplx S;
  const double op[3] = {odd ? nw[0] : old[0], odd ? nw[1] : old[1], odd ? nw[2] : old[2]};
  ev_params(mc, op, odd ? 1.0 : -1.0, C, S, R, shn);
  const double C1 = __shfl_sync(0xffffffffu, C, 0), R1 = __shfl_sync(0xffffffffu, R, 0);
  const double C2 = __shfl_sync(0xffffffffu, C, 1), R2 = __shfl_sync(0xffffffffu, R, 1);
  const cplx S1 = shfl_c(S, 0), S2 = shfl_c(S, 1);
  const double s2 = __shfl_sync(0xffffffffu, shn, 1);
  SitePrep* out = prep + i;
  if (lane < 16) {
    const int r = lane >> 2, c = lane & 3;
    cplx v = cmake(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < 4; ++k) v = cfma(ev_entry(r, k, C1, S1, R1), ev_entry(k, c, C2, S2, R2), v);
    if (r == c) v.x -= 1.0;
    out->delta[lane] = v;
  } else if (lane == 16) {
    EvEntry e;
    e.C = C2; e.Sr = -nw[0] * s2; e.Si = nw[1] * s2; e.R = -nw[2] * s2;
    out->ev = e;
  } else if (lane == 17) {
    // boson action difference (src/action.jl:57-100) without the space-neighbour term
    const int lt_later = (l + 1) % M, lt_earlier = (l - 1 + M) % M;
    const double diff[3] = {nw[0] - old[0], nw[1] - old[1], nw[2] - old[2]};
    const double old_sq = old[0] * old[0] + old[1] * old[1] + old[2] * old[2];
    const double new_sq = nw[0] * nw[0] + nw[1] * nw[1] + nw[2] * nw[2];
    const double sq_diff = new_sq - old_sq;
    const double pow4_diff = new_sq * new_sq - old_sq * old_sq;
    const double* pe = &a.phi[((size_t)N * lt_earlier + i) * 3];
    const double* pl = &a.phi[((size_t)N * lt_later + i) * 3];
    double tdot = 0.0;
    for (int c = 0; c < 3; ++c) tdot += (pl[c] + pe[c]) * diff[c];
    out->diff[0] = diff[0]; out->diff[1] = diff[1]; out->diff[2] = diff[2];
    out->dsA = 1.0 / (mc.dtau * mc.c * mc.c) * (sq_diff - tdot);
    out->dsQ = 4 * sq_diff;
    out->dsB = mc.dtau * (0.5 * mc.r * sq_diff + 0.25 * mc.u * pow4_diff);
  }
}


// Words of a site kept in shared memory: its SitePrep (Delta_i, the proposed
// eV entries, the field difference, the prepared action parts) and the
// Metropolis uniform.
constexpr int kSiteEv = 32, kSiteDiff = 36, kSiteUnif = 44, kSiteWords = 46;
static_assert(sizeof(SitePrep) == 44 * sizeof(double), "SitePrep is read as 44 words");
static_assert(offsetof(SitePrep, ev) == kSiteEv * sizeof(double), "SitePrep.ev");
static_assert(offsetof(SitePrep, diff) == kSiteDiff * sizeof(double), "SitePrep.diff");
static_assert(offsetof(SitePrep, dsA) == (kSiteDiff + 3) * sizeof(double), "SitePrep.dsA");

constexpr int WIN_THREADS = 256;
constexpr int WIN_MAXC = 16;               // CTAs per cluster

// Work split of the 4x4 algebra below: lane = 2 entry + part, so a lane owns
// the real or the imaginary part of one of 16 entries.  An FP64 warp
// instruction costs 64 cycles whatever its active lanes, so this halves the
// instructions of a complex product per entry.
//
// x with its sign flipped where `flip`, on the integer units (a negation that
// is not an operand of an FP64 instruction costs one itself).
__device__ __forceinline__ double flip_sign(double x, bool flip) {
  return __hiloint2double(__double2hiint(x) ^ (flip ? 0x80000000 : 0), __double2loint(x));
}
// Component `part` of a b, as two terms: a.x u + a.y w.
__device__ __forceinline__ void win_uw(cplx b, int part, double& u, double& w) {
  u = part ? b.y : b.x;
  w = flip_sign(part ? b.x : b.y, !part);
}
// Component of sum_k A[r][k] B[k][c] (4x4 blocks, rows of A lda apart, of B 4 apart).
__device__ __forceinline__ double win_mul4(const cplx* A, int lda, const cplx* B, int r, int c, int part) {
  double v0 = 0.0, v1 = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const cplx x = A[r * lda + k];
    double u, w;
    win_uw(B[4 * k + c], part, u, w);
    double& v = k < 2 ? v0 : v1;
    v = fma(x.x, u, v);
    v = fma(x.y, w, v);
  }
  return v0 + v1;
}
// The 12 two-row minors of M = I + Delta (I - g) = (I + Delta) - Delta g
// (src/local_updates.jl:49-55), g a 4x4 block with rows ld apart: minors of
// rows {0, 1} in mn[0..5], of rows {2, 3} in mn[6..11], column pairs (0,1)
// (0,2) (0,3) (1,2) (1,3) (2,3).  One warp; m (16) and mn (12) are its scratch.
__device__ __forceinline__ void win_minors(const cplx* delta, const cplx* g, int ld, cplx* m, cplx* mn, int lane) {
  const int idx = lane >> 1, part = lane & 1, r = idx >> 2, c = idx & 3;
  double v0 = part ? delta[idx].y : delta[idx].x + (r == c ? 1.0 : 0.0), v1 = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const cplx x = delta[4 * r + k];
    double u, w;
    win_uw(g[k * ld + c], part, u, w);
    double& v = k < 2 ? v0 : v1;
    v = fma(-x.x, u, v);
    v = fma(-x.y, w, v);
  }
  reinterpret_cast<double*>(m)[lane] = v0 + v1;
  __syncwarp();
  if (lane < 24) {
    const int mi = lane >> 1, pr = mi < 6 ? 0 : 2, pp = mi < 6 ? mi : mi - 6;
    const int pa = pp < 3 ? 0 : (pp < 5 ? 1 : 2), pb = pp < 3 ? pp + 1 : (pp < 5 ? pp - 1 : 3);
    const cplx e00 = m[4 * pr + pa], e01 = m[4 * pr + pb], e10 = m[4 * pr + 4 + pa], e11 = m[4 * pr + 4 + pb];
    double u, w, u2, w2;
    win_uw(e11, part, u, w);
    win_uw(e10, part, u2, w2);
    const double t1 = fma(e00.y, w, e00.x * u), t2 = fma(e01.y, w2, e01.x * u2);
    reinterpret_cast<double*>(mn)[lane] = t1 - t2;
  }
  __syncwarp();
}
// det M = sum over the column pairs of +-(top minor)(complementary bottom
// minor); real part in lane 0, imaginary part in lane 1.
__device__ __forceinline__ double win_det(const cplx* mn, int lane) {
  const int pp = lane >> 1, part = lane & 1;
  double t = 0.0;
  if (pp < 6) {
    const cplx top = mn[pp];
    double u, w;
    win_uw(mn[11 - pp], part, u, w);
    t = fma(top.y, w, top.x * u);
    t = flip_sign(t, pp == 1 || pp == 4);
  }
#pragma unroll
  for (int o = 8; o > 1; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}
// Component of adj(M)[r][c] (cofactor C[c][r]) of this lane: the 3x3 minor
// expanded along the remaining row of the removed row's pair, over the
// two-row minors of the other pair.
__device__ __forceinline__ double win_adj(const cplx* m, const cplx* mn, int lane) {
  const int idx = lane >> 1, part = lane & 1, rr = idx & 3, cc = idx >> 2;   // removed row, column
  const int other = rr < 2 ? 1 - rr : 5 - rr, base = rr < 2 ? 6 : 0;
  int cols[3];
#pragma unroll
  for (int t = 0; t < 3; ++t) cols[t] = t + (t >= cc ? 1 : 0);
  double d[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int u0 = q == 0 ? cols[1] : cols[0], v0 = q == 2 ? cols[1] : cols[2];
    const int pidx = u0 == 0 ? v0 - 1 : (u0 == 1 ? v0 + 1 : 5);
    const cplx x = m[4 * other + cols[q]];
    double u, w;
    win_uw(mn[base + pidx], part, u, w);
    d[q] = fma(x.y, w, x.x * u);
  }
  return flip_sign((d[0] - d[1]) + d[2], (rr + cc) & 1);
}

// Words that travel between the CTAs of the cluster validate themselves, so
// that no fence stands between writing and reading them: a decision carries
// its step, and a slot of K = M^-1 Delta holds this NaN (which no arithmetic
// produces) until its 8-byte words arrive.
constexpr unsigned long long kWinEmpty = 0x7FF8DEADBEEF0001ull;
// 1 / x by Newton's iteration from a single-precision seed (2^-23, 2^-46,
// then FP64 round-off): four dependent FMAs where the division takes twice
// that; within the single-precision range (recip_range).
__device__ __forceinline__ bool recip_range(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7FF;
  return e >= 1023 - 100 && e <= 1023 + 100;
}
__device__ __forceinline__ double recip_newton(double x) {
  double y = (double)__frcp_rn((float)x);
  y = fma(fma(-x, y, 1.0), y, y);
  return fma(fma(-x, y, 1.0), y, y);
}
// a < b on the integer units (FP64 compares cost FP64 instructions) where the
// bit patterns order like the values: non-negative a and b, b finite
__device__ __forceinline__ bool less_fast(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  if ((x | y) >= 0 && (int)(y >> 52) != 0x7FF) return x < y;
  return a < b;
}
__device__ __forceinline__ bool finite_bits(double x) { return ((__double2hiint(x) >> 20) & 0x7FF) != 0x7FF; }
__device__ __forceinline__ bool zero_bits(double x) { return (__double_as_longlong(x) << 1) == 0; }

__device__ __forceinline__ void named_bar(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The rank-4p factors of a window: G += X Y with
//   X[:, j] = ((G - I)[:, a_j] + sum_{i<j} X[:, i] b_i[a_j]) K_j,
//   Y[j, :] = G[a_j, :] + sum_{i<j} A_i[a_j] Y[i, :]
// (rows of the accepted sites from k_local_window): every row of X and every
// column of Y is an independent recurrence of p steps, taken by 8 SPLIT lanes of a
// warp: 4 components x {real, imaginary} x SPLIT shares of the sum over i.  At
// the end each vector is cut into the BF16 slices of the flush.
// Bound: FP64 issue, 8 (4p)^2 / 2 multiply-adds per vector.
struct FacLane {
  int part, q, sp, v;   // this lane's component, share of the sum and vector of its warp
};
template <int SPLIT>
__device__ __forceinline__ FacLane fac_lane() {
  const int lane = threadIdx.x & 31;
  return {lane & 1, (lane >> 1) & 3, (lane >> 3) % SPLIT, lane / (8 * SPLIT)};
}
// Step j of one vector x (4 p entries; entry 4 j + q holds g on entry): cj the
// blocks of the terms i < j, [i][c][q]; kj the block K_j (X only); t scratch of 4.
template <int SPLIT>
__device__ __forceinline__ void fac_step(const FacLane& f, cplx* x, int j, const cplx* cj, const cplx* kj, cplx* ts) {
  double t0 = 0.0, t1 = 0.0;
  if (f.sp == 0) t0 = f.part ? x[4 * j + f.q].y : x[4 * j + f.q].x;
#pragma unroll 1
  for (int i = f.sp; i < j; i += SPLIT) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const cplx xv = x[4 * i + c];
      double u, w;
      win_uw(cj[16 * i + 4 * c + f.q], f.part, u, w);
      t0 = fma(xv.x, u, t0);
      t1 = fma(xv.y, w, t1);
    }
  }
  double t = t0 + t1;
#pragma unroll
  for (int o = 8; o < 8 * SPLIT; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (kj) {
    if (f.sp == 0) reinterpret_cast<double*>(&ts[f.q])[f.part] = t;
    __syncwarp();
    double r0 = 0.0, r1 = 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const cplx tv = ts[c];
      double u, w;
      win_uw(kj[4 * c + f.q], f.part, u, w);
      r0 = fma(tv.x, u, r0);
      r1 = fma(tv.y, w, r1);
    }
    t = r0 + r1;
  }
  __syncwarp();
  if (f.sp == 0) reinterpret_cast<double*>(x + 4 * j + f.q)[f.part] = t;
  __syncwarp();
}
// block element e (4 c + q of the step) of term i in step j: X takes b_i[a_j],
// Y the transpose of A_i[a_j]; si, sj: the sites' places in the window
__device__ __forceinline__ cplx fac_coef(const DelayedArgs& d, int side, int j, int i, int sj, int si, int e) {
  const int c = e >> 2, q = e & 3;
  return side == 0 ? ldcg_c(&d.wrow[((size_t)i * 4 + c) * (4 * WIN_MAX) + 4 * sj + q])
                   : ldcg_c(&d.wrow[((size_t)j * 4 + q) * (4 * WIN_MAX) + 4 * si + c]);
}
// entry q of step j before the recurrence, of vector v
__device__ __forceinline__ cplx fac_entry(const LocalUpdateArgs& a, int side, int site, int q, int v) {
  const int n = a.mc.n, ai = site + q * a.mc.N;
  cplx g = side == 0 ? ldcg_c(&a.G[(size_t)ai * n + v]) : ldcg_c(&a.G[(size_t)v * n + ai]);
  if (side == 0 && ai == v) g.x -= 1.0;
  return g;
}
// a warp's VPW finished vectors from v0 on
template <int VPW>
__device__ __forceinline__ void fac_finish(const DelayedArgs& d, int side, int v0, int p, const cplx* xs, int ldx) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int u = 0; u < VPW; ++u) {
    const cplx* xv = xs + u * ldx;
    oz_slice_vec(d.sl, side, v0 + u, 4 * p, [&](int k) { return xv[k]; }, lane);
  }
}

// The factors as a launch of their own, after the window (chains that share the
// GPU).  SPLIT grows as n falls, so that small lattices still fill the
// sub-partitions.
constexpr int FAC_THREADS = 128;
template <int SPLIT>
__global__ void __launch_bounds__(FAC_THREADS) k_local_factors(LocalUpdateArgs a, DelayedArgs d) {
  const int p = __ldcg(&d.state[1]);
  if (p == 0) return;   // uniform over the grid
  constexpr int VPW = 4 / SPLIT, VPC = VPW * (FAC_THREADS / 32);
  const int side = blockIdx.y, v0 = blockIdx.x * VPC;   // side 0: rows of X, 1: columns of Y
  extern __shared__ double4_16a smem_fac[];
  cplx* coef = reinterpret_cast<cplx*>(smem_fac);       // (p (p - 1) / 2, 4, 4): [c][q] of step j, term i < j
  cplx* kk = coef + (size_t)8 * p * (p - 1);            // (p, 4, 4) K_j (X)
  const int ldx = 4 * d.k + 1;
  cplx* xs = kk + 16 * p;                               // (VPC, ldx) the vectors
  __shared__ cplx s_t[VPC][4];
  __shared__ int s_site[WIN_MAX];
  const int tid = threadIdx.x, wid = tid >> 5;
  const int base = __ldcg(&d.state[3]);
  if (tid < p) s_site[tid] = __ldcg(&d.wsite[tid]);
  __syncthreads();
#pragma unroll 4
  for (int e = tid; e < 8 * p * (p - 1); e += FAC_THREADS) {
    // pair index (j, i): j (j - 1) / 2 + i
    const int pr = e >> 4;
    int j = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)pr)) * 0.5f);
    while (j * (j - 1) / 2 > pr) --j;
    while ((j + 1) * j / 2 <= pr) ++j;
    const int i = pr - j * (j - 1) / 2;
    coef[e] = fac_coef(d, side, j, i, s_site[j], s_site[i], e & 15);
  }
  if (side == 0)
    for (int e = tid; e < 16 * p; e += FAC_THREADS) kk[e] = ldcg_c(&d.wk[e]);
#pragma unroll 4
  for (int e = tid; e < 4 * p * VPC; e += FAC_THREADS) {
    const int v = side == 0 ? e % VPC : e / (4 * p), jq = side == 0 ? e / VPC : e - v * 4 * p;
    xs[v * ldx + jq] = fac_entry(a, side, base + s_site[jq >> 2], jq & 3, v0 + v);
  }
  __syncthreads();
  const FacLane f = fac_lane<SPLIT>();
  const int v = wid * VPW + f.v;
  for (int j = 0; j < p; ++j)
    fac_step<SPLIT>(f, xs + v * ldx, j, coef + (size_t)8 * j * (j - 1), side == 0 ? kk + 16 * j : nullptr, s_t[v]);
  fac_finish<VPW>(d, side, v0 + wid * VPW, p, xs + wid * VPW * ldx, ldx);
}

// The factors beside the window (a chain that has the GPU to itself): a CTA of
// a follower cluster takes step j of its VPC = 4 WARPS / SPLIT vectors as soon as
// the window's cluster has published the j-th acceptance, so that only the last
// step and the slicing are left when the window is decided.  One warp per CTA
// polls: a poll of every warp keeps the word's L2 slice busy.
template <int SPLIT, int WARPS>
__device__ void fac_follow(const LocalUpdateArgs& a, const DelayedArgs& d, int first, int blk, cplx* smem) {
  constexpr int VPW = 4 / SPLIT, VPC = VPW * WARPS, T = 32 * WARPS;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, n = a.mc.n;
  const int ctas = (n + VPC - 1) / VPC, side = blk < ctas ? 0 : 1;
  if (blk >= 2 * ctas) return;
  const int v0 = (blk - side * ctas) * VPC, nv = min(VPC, n - v0);   // nv: a multiple of 4
  const int ldx = 4 * d.k + 1;
  cplx* xs = smem;                          // (VPC, ldx)
  cplx* cj = xs + VPC * ldx;                // (WIN_MAX, 4, 4)
  cplx* kj = cj + 16 * WIN_MAX;             // (4, 4)
  cplx* ts = kj + 16;                       // (VPC, 4)
  int* sites = reinterpret_cast<int*>(ts + 4 * VPC);   // (WIN_MAX) and the word of the step
  const FacLane f = fac_lane<SPLIT>();
  const int v = wid * VPW + f.v;
  int j = 0;
  for (;; ++j) {
    if (wid == 0) {
      int w = 0;
      bool here = false;
      for (int it = 0; it < kClusterPolls && !here; ++it) {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w) : "l"(d.wflag + j) : "memory");
        here = __all_sync(0xffffffffu, (w >> 9) == first + 1);
      }
      __threadfence();
      if (lane == 0) sites[WIN_MAX] = here ? w : -1;
    }
    named_bar(1, T);   // also: the coefficients of the step before are read
    const int w = sites[WIN_MAX];
    if (w < 0) {
      if (tid == 0) atomicOr(a.err, DQMC_KERR_BARRIER_TIMEOUT);
      return;
    }
    if (!(w & 256)) break;   // no further acceptance
    const int sj = w & 255;
    if (tid == 0) sites[j] = sj;
    for (int e = tid; e < 16 * j; e += T) cj[e] = fac_coef(d, side, j, e >> 4, sj, sites[e >> 4], e & 15);
    if (tid < 4 * nv) {
      const int u = side == 0 ? tid % nv : tid >> 2, q = side == 0 ? tid / nv : tid & 3;
      xs[u * ldx + 4 * j + q] = fac_entry(a, side, first + sj, q, v0 + u);
    }
    if (side == 0 && tid >= T - 16) kj[tid - (T - 16)] = ldcg_c(&d.wk[16 * j + tid - (T - 16)]);
    named_bar(1, T);
    if (wid * VPW < nv) fac_step<SPLIT>(f, xs + v * ldx, j, cj, side == 0 ? kj : nullptr, ts + 4 * v);
  }
  if (j > 0 && wid * VPW < nv) fac_finish<VPW>(d, side, v0 + wid * VPW, j, xs + wid * VPW * ldx, ldx);
}

// Vectors of a follower CTA: the fewest that keep the followers within 7
// clusters of 16 CTAs.  With the window's own these have a GPC each; an eighth
// shares its SMs with another (n > 896), which doubles the time of its steps.
__host__ __device__ constexpr int fac_vpc(int n) { return n <= 224 ? 4 : (n <= 448 ? 8 : 16); }
// and their words of shared memory
__host__ __device__ constexpr int fac_follow_smem(int n, int k) {
  return fac_vpc(n) * (4 * k + 1) + 16 * WIN_MAX + 16 + 4 * fac_vpc(n) + WIN_MAX / 4 + 1;
}

// Decides the window of sites state[0] .. state[0] + W - 1 (fewer at the
// slice's end; it also ends once d.k sites are accepted) on one cluster of C
// CTAs.  Site s of the window (0-based) belongs to CTA s mod C, which holds its
// 4 rows of the window's block of G (4 x 4W, column 4 s' + flavour).
//
// The next C undecided sites are evaluated at once, one per CTA, each as if
// the ones before it were rejected; the first accepted one, in order, is the
// chain's next acceptance, and the ones before it are rejected for good.  The
// chain therefore costs one step per accepted site (and none per rejected
// one).  Roles of the warps in a step:
//   0  det M and the decision;          1  K = M^-1 Delta, pushed to all CTAs;
//   2  exp(-dS), then 1 / det;          3  publishes the decision, polls all CTAs';
//   4-7  read the accepted site's rows b = G[a, .] from its owner;
//   0, 1  A = G[r, a] K of the own undecided rows, then the diagonal block of
//         the next candidate, with which they start its evaluation at once;
//   3-7  the rest of G[r, .] += A b, beside that evaluation.
// Rows of decided sites stay as they were when decided.
//
// For the factors of the accepted sites a_1 .. a_p (in order) the kernel leaves
// K_j = M_j^-1 Delta_j and the rows of a_j as they were when it was accepted: in
// the columns of a later site a_l they are b_j[a_l] = G_{j-1}[a_j, a_l], in those of
// an earlier one A_i[a_j] = (G_{i-1} - I)[a_j, a_i] K_i (which takes the place of the
// column once it is no longer needed).  With follower clusters (gridDim.x > C)
// those form the factors at the same time, acceptance by acceptance.
//
// Bound: the chain of dependent FP64 operations of a step, about 100 cycles
// each (64 to issue one).  The kernel this replaces formed all n rows and
// columns of each acceptance before the next decision and took 7.6 us per
// accepted and 3.6 us per rejected site at n = 1024.
__global__ void __launch_bounds__(WIN_THREADS) k_local_window(LocalUpdateArgs a, DelayedArgs d, int W, int C) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const ModelConst& mc = a.mc;
  const int N = mc.N, n = mc.n, L = mc.L;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if ((int)cl.num_blocks() != C) {   // not the clusters that shared memory was sized for
    if (tid == 0) atomicOr(a.err, DQMC_KERR_BAD_SHAPE);
    return;
  }
  const int first = __ldcg(&d.state[0]);
  extern __shared__ double4_16a smem_win[];
  const int followers = (int)gridDim.x - C;   // their CTAs, in clusters after the window's
  if (first >= N) {   // slice done (uniform over the grid): nothing for the flush either
    if (blockIdx.x == 0 && tid == 0) d.state[1] = 0;   // read by nobody in this launch
    return;
  }
  // With followers, the first cluster to start takes the window: whoever waits
  // then waits for a cluster that runs, in whatever order clusters are placed.
  // Every cluster loads the window meanwhile.
  __shared__ int s_ticket;
  int ticket = 0;
  if (followers > 0) {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    if (rank == 0 && tid == 0) {
      ticket = atomicAdd(d.arrive + 1, 1);
      // after a timeout the arrivals are those of the window that timed out, until
      // the next preparation: nobody starts (decided once for the cluster)
      if (__ldcg(a.err) & DQMC_KERR_BARRIER_TIMEOUT) ticket = -1;
    }
  }
  const int we = min(W, N - first);                       // sites of this window
  const int owned = rank < we ? (we - rank + C - 1) / C : 0;   // sites rank + t C
  const int own_max = (W + C - 1) / C;
  const int LD = 4 * W + 1;
  cplx* Gs = reinterpret_cast<cplx*>(smem_win);           // (4 own_max, LD)
  cplx* brow = Gs + (size_t)4 * own_max * LD;             // (4, 4W) rows of the accepted site
  cplx* As = brow + 16 * W;                               // (4 own_max, 4): G[r, a] M^-1 Delta
  double* site = reinterpret_cast<double*>(As + 16 * own_max);   // (own_max, kSiteWords)
  double* prop = site + (size_t)own_max * kSiteWords;     // (W, 3) proposals
  double* phis = prop + 3 * W + (W & 1);                  // (3, N) field of the slice
  __shared__ cplx s_m[2][16], s_mn[2][12], s_adj[16], s_g[2][16];
  __shared__ cplx s_k[3][WIN_MAXC][16];                   // K of the accepting candidates, by step mod 3 and owner
  __shared__ int s_pub[2][WIN_MAXC];                      // (step + 1) << 1 | accepted, by parity (both written by the owners)
  __shared__ double s_exp[2], s_det[2];
  __shared__ cplx s_inv;
  __shared__ int s_acc[WIN_MAX], s_fin[2], s_dec[2], s_flag[2];
  if (tid < 2 * WIN_MAXC) s_pub[0][tid] = 0;
  for (int e = tid; e < 3 * 2 * WIN_MAXC * 16; e += WIN_THREADS)
    reinterpret_cast<unsigned long long*>(s_k)[e] = kWinEmpty;
  for (int e = tid; e < owned * 16 * we; e += WIN_THREADS) {
    const int rr = e / (4 * we), c = e - rr * 4 * we, t = rr >> 2, r = rr & 3;
    Gs[(size_t)rr * LD + c] =
        ldcg_c(&a.G[(size_t)(first + (c >> 2) + (c & 3) * N) * n + first + rank + t * C + r * N]);
  }
  for (int e = tid; e < owned * kSiteWords; e += WIN_THREADS) {
    const int t = e / kSiteWords, k = e - t * kSiteWords, gi = first + rank + t * C;
    site[e] = k < 44 ? __ldcg(reinterpret_cast<const double*>(d.prep + gi) + k) : (k == kSiteUnif ? a.unif[gi] : 0.0);
  }
  for (int e = tid; e < 3 * we; e += WIN_THREADS) prop[e] = a.delta[3 * first + e];
  for (int e = tid; e < 3 * N; e += WIN_THREADS) phis[e] = __ldcg(&a.phi[(size_t)3 * N * a.slice0 + e]);
  if (followers > 0) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // every CTA of the cluster runs
    if (rank == 0 && tid < C) *cl.map_shared_rank(&s_ticket, tid) = __shfl_sync((1u << C) - 1, ticket, 0);
  }
  cl.sync();   // also: every CTA of the cluster runs before its shared memory is written remotely
  if (followers > 0 && s_ticket < 0) {
    if (blockIdx.x == 0 && tid == 0) d.state[1] = 0;
    return;
  }
  if (followers > 0 && s_ticket > 0) {
    if (tid == 0) {   // the state has been read: the window may advance it
      __threadfence();
      atomicAdd(d.arrive, 1);
    }
    const int blk = (s_ticket - 1) * C + rank, vpc = fac_vpc(n);
    cplx* sm = reinterpret_cast<cplx*>(smem_win);
    if (vpc == 4) {
      if (wid < 4) fac_follow<4, 4>(a, d, first, blk, sm);
    } else if (vpc == 8) {
      fac_follow<4, 8>(a, d, first, blk, sm);
    } else {
      fac_follow<2, 8>(a, d, first, blk, sm);
    }
    return;
  }

  const int part = lane & 1, r = lane >> 3, c = (lane >> 1) & 3;   // this lane's component of a 4x4 block
  int cur = 0, p = 0;
  bool ok = true, fresh = true;   // fresh: the candidate's diagonal block is to be read from Gs
  // a CTA leaves the loop once all its sites are decided; every CTA in it has a
  // candidate, publishes at every step and waits for all of them, so none can
  // be two steps ahead of another and two buffers by step parity suffice.  A
  // slot of K is emptied two steps after its use: every candidate's decision
  // of the next step has then been seen, and with it the K it pushed (only
  // accepting candidates push, and those either are waited for or stay in the
  // loop).
  for (int step = 0; owned > 0 && cur < we && p < d.k; ++step) {
    const int par = step & 1, kslot = step % 3;
    const int sc = cur + (rank - cur % C + C) % C;   // this CTA's candidate: its first undecided site
    const int t = sc / C;
    const double* sw = site + (size_t)t * kSiteWords;
    const cplx* delta = reinterpret_cast<const cplx*>(sw);
    const int ncand = min(C, we - cur);
    double kv = 0.0;   // warp 1: this lane's component of K
    if (wid < 2 && fresh) {
      reinterpret_cast<double*>(s_g[wid])[lane] =
          reinterpret_cast<const double*>(Gs + (size_t)(4 * t + r) * LD + 4 * sc + c)[part];
      __syncwarp();
    }
    if (wid == 0) {
      win_minors(delta, s_g[0], 4, s_m[0], s_mn[0], lane);
      const double det = win_det(s_mn[0], lane);
      if (lane < 2) s_det[lane] = det;
      __syncwarp();
      named_arrive(4, 64);   // det for warp 2
      named_bar(1, 64);      // exp(-dS) from warp 2
      const double dx = __shfl_sync(0xffffffffu, det, 0), dy = __shfl_sync(0xffffffffu, det, 1);
      const double ex = s_exp[par];
      const double pa = ex * dx;
      const bool bad = !finite_bits(dx) || !finite_bits(dy) || (zero_bits(dx) && zero_bits(dy));
      const bool ac = !bad && (less_fast(1.0, pa) || less_fast(sw[kSiteUnif], pa));   // src/local_updates.jl:20-30
      if (lane == 0) s_flag[par] = (ac ? 1 : 0) | (bad ? 2 : 0);
      __syncwarp();
      named_arrive(3, 96);   // decision for warps 1 and 3
    } else if (wid == 1) {
      win_minors(delta, s_g[1], 4, s_m[1], s_mn[1], lane);
      reinterpret_cast<double*>(s_adj)[lane] = win_adj(s_m[1], s_mn[1], lane);
      __syncwarp();
      const double kp = win_mul4(s_adj, 4, delta, r, c, part);
      const double o = __shfl_xor_sync(0xffffffffu, kp, 1);
      named_bar(5, 64);      // 1 / det from warp 2
      const cplx inv = s_inv;
      kv = fma(o, flip_sign(inv.y, !part), kp * inv.x);
      named_bar(3, 96);
      if (s_flag[par] & 1)
        for (int q = 0; q < C; ++q)
          st_cluster(cl.map_shared_rank(reinterpret_cast<double*>(s_k[kslot][rank]) + lane, q),
                     (unsigned long long)__double_as_longlong(kv));
    } else if (wid == 2) {
      // boson action difference: prepared part + space-neighbour coupling;
      // lanes 0-2 sum the neighbours' component c = lane, lane 0 takes the rest
      const int gi = first + sc, y = gi % L, x = gi / L;
      const int nbs[4] = {(y + 1) % L + L * x, y + L * ((x + 1) % L), (y - 1 + L) % L + L * x,
                          y + L * ((x - 1 + L) % L)};
      double os = 0.0;
      if (lane < 3)
        for (int q = 0; q < 4; ++q) os = os + phis[3 * nbs[q] + lane];
      const double os1 = __shfl_sync(0xffffffffu, os, 1), os2 = __shfl_sync(0xffffffffu, os, 2);
      if (lane == 0) {
        const double osc[3] = {os, os1, os2};
        double sdot = 0.0;
        for (int q = 0; q < 3; ++q) sdot += osc[q] * sw[kSiteDiff + q];
        double dS = sw[kSiteDiff + 3];
        dS += 0.5 * mc.dtau * (sw[kSiteDiff + 4] - 2.0 * sdot);
        dS += sw[kSiteDiff + 5];
        s_exp[par] = exp(-dS);
      }
      __syncwarp();
      named_arrive(1, 64);
      named_bar(4, 64);
      if (lane == 0) {
        const double dx = s_det[0], dy = s_det[1];
        const double d2 = fma(dx, dx, dy * dy);
        if (recip_range(d2)) {
          const double rd = recip_newton(d2);
          s_inv = cmake(dx * rd, flip_sign(dy * rd, true));
        } else {   // also where the square leaves the range of double
          s_inv = cdiv(cmake(1.0, 0.0), cmake(dx, dy));
        }
      }
      __syncwarp();
      named_arrive(5, 64);
    } else if (wid == 3) {
      // empty the K slots of two steps ago; the own rows are complete (barrier 6
      // below): order both before the decision
      for (int e = lane; e < 2 * WIN_MAXC * 16; e += 32)
        reinterpret_cast<unsigned long long*>(s_k[(step + 1) % 3])[e] = kWinEmpty;
      __syncwarp();
      fence_release_shared();
      named_bar(3, 96);
      const int flag = s_flag[par];
      if (lane < C) st_cluster(cl.map_shared_rank(&s_pub[par][rank], lane), (step + 1) << 1 | (flag & 1));
      // the first accepted candidate in site order (the same in every CTA) once
      // all candidates are published; -2: gave up waiting
      int acc3 = -2;
      for (int it = 0; it < kClusterPolls; ++it) {
        int v = (step + 1) << 1;
        if (lane < ncand) v = ld_poll(&s_pub[par][(cur + lane) % C]);
        if (__all_sync(0xffffffffu, v >> 1 == step + 1)) {
          const unsigned hit = __ballot_sync(0xffffffffu, v & 1);
          acc3 = hit ? cur + __ffs(hit) - 1 : -1;
          break;
        }
      }
      fence_acquire_shared();
      if (lane == 0) s_dec[par] = acc3;
    }
    __syncthreads();
    const int acc = s_dec[par];
    if (acc == -2) {
      ok = false;
      break;
    }
    // orders warp 1's K words before this CTA's next decision (about 950 cycles,
    // beside the reads of the accepted site's rows)
    if (wid == 3) fence_cluster();
    const int last = acc >= 0 ? acc : cur + ncand - 1;   // sites cur .. last are decided
    if (sc <= last && wid == 3 && lane == 0) {
      const int gi = first + sc, flag = s_flag[par];
      if (flag & 2) atomicOr(a.err, DQMC_KERR_NONFINITE);
      if (a.acc_out) a.acc_out[gi] = (uint8_t)(flag & 1);
      if (a.det_out) a.det_out[gi] = cmake(s_det[0], s_det[1]);
      if (a.pacc_out) a.pacc_out[gi] = s_exp[par] * s_det[0];
    }
    cur = last + 1;
    const int t0 = rank > last ? 0 : (last - rank) / C + 1;   // own undecided sites t0 .. owned - 1
    fresh = true;
    if (acc < 0) {
      if (t0 >= owned) break;
      __syncthreads();   // s_det, s_flag read
      continue;
    }
    const int owner = acc % C, ta = acc / C;
    if (rank == owner) {
      // K and the rows of the accepted site for the factors, published by warp 4
      if (wid == 1) {
        reinterpret_cast<double*>(d.wk + 16 * p)[lane] = kv;
        __syncwarp();
        named_arrive(7, 160);
      } else if (wid >= 4) {
        const cplx* src = Gs + (size_t)(4 * ta + wid - 4) * LD;
        cplx* dst = d.wrow + ((size_t)p * 4 + wid - 4) * (4 * WIN_MAX);
        for (int cc = lane; cc < 4 * we; cc += 32) dst[cc] = src[cc];
        __syncwarp();
        if (wid > 4) {
          named_arrive(7, 160);
        } else {
          named_bar(7, 160);
          if (lane == 0) {
            __threadfence();
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(d.wflag + p), "r"((first + 1) << 9 | 256 | acc)
                         : "memory");
          }
          __syncwarp();
        }
      }
    }
    if (wid == 2) {
      // field, interaction table, order of acceptances
      const int gi = first + acc;
      if (lane < 3) {
        const double v = phis[3 * gi + lane] + prop[3 * acc + lane];
        phis[3 * gi + lane] = v;
        if (rank == owner) a.phi[((size_t)N * a.slice0 + gi) * 3 + lane] = v;
      } else if (lane == 3) {
        s_acc[p] = acc;
        if (rank == owner) d.wexp[p] = s_exp[par];
      } else if (lane == 4 && rank == owner && a.evtab) {
        const double* se = site + (size_t)ta * kSiteWords + kSiteEv;
        EvEntry ev;
        ev.C = se[0]; ev.Sr = se[1]; ev.Si = se[2]; ev.R = se[3];
        reinterpret_cast<EvEntry*>(a.evtab)[(size_t)N * a.slice0 + gi] = ev;
      }
      __syncwarp();
    }
    ++p;
    if (t0 >= owned) break;
    if (wid != 2) {
      // ---- apply the acceptance to the own undecided rows (7 warps) ----
      const int left = owned - t0, cols = 4 * (we - acc - 1), c0 = 4 * (acc + 1);
      const int s0 = rank + t0 * C;   // the next candidate
      double gv = 0.0;                // warps 0, 1: this lane's component of its diagonal block
      if (wid < 2) {
        gv = reinterpret_cast<const double*>(Gs + (size_t)(4 * t0 + r) * LD + 4 * s0 + c)[part];
        const cplx* k = s_k[kslot][owner];
        bool here = false;
        for (int it = 0; it < kClusterPolls && !here; ++it) {
          const int w0 = ld_poll(reinterpret_cast<const int*>(k) + 2 * lane);
          const int w1 = ld_poll(reinterpret_cast<const int*>(k) + 2 * lane + 1);
          here = __all_sync(0xffffffffu, w0 != (int)(kWinEmpty & 0xffffffffu) || w1 != (int)(kWinEmpty >> 32));
        }
        fence_acquire_shared();
        __syncwarp();
        ok = ok && here;
        for (int ts = t0 + wid; ts < owned; ts += 2) {
          const double v = win_mul4(Gs + (size_t)4 * ts * LD + 4 * acc, LD, k, r, c, part);
          reinterpret_cast<double*>(As + 16 * ts)[lane] = v;
          __syncwarp();
          reinterpret_cast<double*>(Gs + (size_t)(4 * ts + r) * LD + 4 * acc + c)[part] = v;
        }
      } else if (wid >= 4) {
        const int q = wid - 4;
        const cplx* src = cl.map_shared_rank(Gs + (size_t)(4 * ta + q) * LD + c0, owner);
        cplx* dst = brow + q * 4 * W + c0;
        for (int cc = lane; cc < cols; cc += 64) {
          const bool two = cc + 32 < cols;
          const cplx x0 = src[cc], x1 = two ? src[cc + 32] : cmake(0.0, 0.0);
          dst[cc] = x0;
          if (two) dst[cc + 32] = x1;
        }
      }
      named_bar(2, WIN_THREADS - 32);
      if (wid < 2) {
        // G[row, cc] += sum_q A[row][q] b[q][cc]
        const cplx* ar = As + 4 * (4 * t0 + r);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double u, w;
          win_uw(brow[q * 4 * W + 4 * s0 + c], part, u, w);
          gv = fma(ar[q].x, u, gv);
          gv = fma(ar[q].y, w, gv);
        }
        reinterpret_cast<double*>(s_g[wid])[lane] = gv;
        __syncwarp();
      } else {
        // one entry per lane: two independent chains (real, imaginary) hide the
        // FP64 latency that one leaves exposed
        const float icols = 1.0f / (float)cols;
        for (int e = tid - 96; e < 4 * left * cols; e += 160) {
          const int rr = (int)(((float)e + 0.5f) * icols), cc = c0 + e - rr * cols, row = 4 * t0 + rr;
          const cplx* ar = As + 4 * row;
          cplx v = Gs[(size_t)row * LD + cc];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const cplx x = ar[q], y = brow[q * 4 * W + cc];
            v.x = fma(x.x, y.x, v.x);
            v.y = fma(x.x, y.y, v.y);
            v.x = fma(-x.y, y.y, v.x);
            v.y = fma(x.y, y.x, v.y);
          }
          Gs[(size_t)row * LD + cc] = v;
        }
        named_bar(6, 160);   // warps 3-7: the own rows are complete
      }
    }
    fresh = false;
  }
  if (!ok) atomicOr(a.err, DQMC_KERR_BARRIER_TIMEOUT);
  const int lastr = (we - 1) % C;   // has seen all decisions
  if (followers > 0 && rank == lastr && tid == 0)   // no further acceptance
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(d.wflag + p), "r"((first + 1) << 9) : "memory");
  if (wid == 2 && lane == 0) {
    s_fin[0] = p;
    s_fin[1] = cur;
  }
  cl.sync();   // every CTA is done; the owner of the last site has seen all decisions
  p = *cl.map_shared_rank(&s_fin[0], lastr);
  cur = *cl.map_shared_rank(&s_fin[1], lastr);
  __syncthreads();
  if (rank != lastr) {
    for (int e = tid; e < p; e += WIN_THREADS) s_acc[e] = cl.map_shared_rank(&s_acc[0], lastr)[e];
  }
  cl.sync();   // no shared memory is read remotely any more
  // ---- the round's state ----
  if (rank == 0 && wid == 0) {
    if (lane < p) d.wsite[lane] = s_acc[lane];
    int late = __ldcg(a.err) & DQMC_KERR_BARRIER_TIMEOUT;   // of any CTA: before the barriers above
    if (lane == 0 && followers > 0) {
      // the followers have read the state (bounded wait)
      bool here = false;
      for (int it = 0; it < kClusterPolls && !here; ++it) here = *(volatile int*)d.arrive == followers;
      if (!here) {
        atomicOr(a.err, DQMC_KERR_BARRIER_TIMEOUT);
        late = 1;
      }
      if (!late) {
        d.arrive[0] = 0;
        d.arrive[1] = 0;
      }
    }
    late = __shfl_sync(0xffffffffu, late, 0);
    if (late) {   // a follower may still arrive or read the state: both stay as they are, and the flush has nothing to do
      if (lane == 0) d.state[1] = 0;
      return;
    }
    // the tracked action: -log(exp(-dS)) of the accepted sites, added in order
    const double lg = lane < p ? -log(__ldcg(&d.wexp[lane])) : 0.0;
    double act = lane == 0 ? *a.action : 0.0;
    for (int q = 0; q < p; ++q) {
      const double v = __shfl_sync(0xffffffffu, lg, q);
      if (lane == 0) act += v;
    }
    if (lane == 0) {
      d.state[0] = first + cur;
      d.state[1] = p;
      d.state[3] = first;
      if (p > 0) {
        *a.action = act;
        *a.n_acc += p;
      }
    }
  }
}

// Condition of the graph's WHILE node that repeats [delayed round, flush]:
// one more round while sites of the slice remain, at most max_rounds rounds
// per slice (state[2] counts them from the prepare kernel on), and none after
// an error bit is set.  rounds_total counts every round run this way.
__global__ void k_round_cond(cudaGraphConditionalHandle hc, int* state, int N, int max_rounds, const int* err,
                             unsigned long long* rounds_total) {
  if (threadIdx.x == 0) {
    const int it = state[2] + 1;
    state[2] = it;
    const bool more = it < max_rounds && __ldcg(&state[0]) < N && __ldcg(err) == 0;
    cudaGraphSetConditional(hc, more ? 1u : 0u);
    *rounds_total += 1ull;
  }
}

}  // namespace

cudaError_t launch_round_cond(cudaGraphConditionalHandle hc, int* state, int N, int max_rounds, const int* err,
                              unsigned long long* rounds_total, cudaStream_t st) {
  k_round_cond<<<1, 32, 0, st>>>(hc, state, N, max_rounds, err, rounds_total);
  return cudaGetLastError();
}

static size_t local_smem_bytes(int N) {
  return (size_t)N * (16 * sizeof(cplx) + sizeof(EvEntry)) + (size_t)3 * N * sizeof(double);
}

cudaError_t launch_local_prepare(const LocalUpdateArgs& a, SitePrep* prep, int* state, int* wflag, cudaStream_t st) {
  k_local_prepare<<<(a.mc.N + 3) / 4, 128, 0, st>>>(a, prep, state, wflag);
  return cudaGetLastError();
}

static size_t window_smem(int N, int W, int C) {
  const size_t own = (size_t)(W + C - 1) / C;
  return (4 * own * (4 * W + 1) + 16 * W + 16 * own) * sizeof(cplx) +
         (own * kSiteWords + 3 * W + (W & 1) + 3 * N) * sizeof(double);
}

static cudaLaunchConfig_t window_config(cudaLaunchAttribute* attr, int C, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(WIN_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Cluster size of the window kernel on the current device: 16 CTAs where the
// device can schedule one (a non-portable size), else 8.
static cudaError_t window_cluster(int* C) {
  static std::mutex mu;
  static int cached[64] = {};
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == 0) {
    const void* fn = (const void*)k_local_window;
    if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1); e != cudaSuccess)
      return e;
    for (int c = WIN_MAXC; c >= 8 && cached[dev] == 0; c /= 2) {
      const size_t smem = window_smem(256, WIN_MAX, c);   // the largest lattice and window
      if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
          e != cudaSuccess)
        return e;
      cudaLaunchAttribute attr[1];
      const cudaLaunchConfig_t cfg = window_config(attr, c, smem, nullptr);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        clusters = 0;
      }
      if (clusters >= 1) cached[dev] = c;
    }
    if (cached[dev] == 0) return cudaErrorNotSupported;
    // 8-CTA clusters (batched chains) hold up to four sites per CTA; the followers of the deepest windows
    const size_t most = std::max(window_smem(256, WIN_MAX, 8), (size_t)fac_follow_smem(1024, 64) * sizeof(cplx));
    if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        e != cudaSuccess)
      return e;
  }
  *C = cached[dev];
  return cudaSuccess;
}

// Sites of a window: k, so that the acceptances of most windows fit their round; twice
// as many for k < 8, where rejected sites would leave rounds nearly empty (L = 16
// mixed, depth 2, 20 calls: 128 ms with a round per 2 acceptances, 140 with a window
// of 2 sites), and at most one site per CTA of the cluster is no more work.
int local_window_sites(int k) { return k < 8 ? 2 * k : (k < WIN_MAX ? k : WIN_MAX); }

// Follower clusters of a window launch.
static int follower_clusters(int n, int C) { return (2 * ((n + fac_vpc(n) - 1) / fac_vpc(n)) + C - 1) / C; }

cudaError_t launch_local_window(const LocalUpdateArgs& a, const DelayedArgs& d, cudaStream_t st, bool shared,
                                bool follow) {
  int C = 0;
  if (cudaError_t e = window_cluster(&C); e != cudaSuccess) return e;
  // 16 free SMs in one GPC are rare beside other chains' QRs, which fill their SMs:
  // with the LU panels likewise, 16 chains of L = 6 .. 12 484 -> 458 ms, 8 of L = 16
  // 899 -> 772 ms per 40 calls
  if (shared && C > 8) C = 8;
  const int W = local_window_sites(d.k);
  size_t smem = window_smem(a.mc.N, W, C);
  cudaLaunchAttribute attr[1];
  if (follow) {
    const size_t fs = (size_t)fac_follow_smem(a.mc.n, d.k) * sizeof(cplx);
    if (fs > smem) smem = fs;
  }
  cudaLaunchConfig_t cfg = window_config(attr, C, smem, st);
  if (follow) cfg.gridDim = dim3(C * (1 + follower_clusters(a.mc.n, C)));
  return cudaLaunchKernelEx(&cfg, k_local_window, a, d, W, C);
}

bool local_window_follows(int n, int k) {
  int C = 0;
  if (window_cluster(&C) != cudaSuccess) return false;
  const int W = local_window_sites(k);
  size_t smem = window_smem(n / 4, W, C);
  const size_t fs = (size_t)fac_follow_smem(n, k) * sizeof(cplx);
  if (fs > smem) smem = fs;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = window_config(attr, C, smem, nullptr);
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, (const void*)k_local_window, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return clusters >= 1 + follower_clusters(n, C);
}

cudaError_t launch_local_factors(const LocalUpdateArgs& a, const DelayedArgs& d, int sm_count, cudaStream_t st) {
  const int n = a.mc.n, W = local_window_sites(d.k);
  // lanes per vector: 2 n vectors of 8 split lanes on 4 sub-partitions per SM, one warp each
  const int split = n <= 2 * sm_count ? 4 : n <= 4 * sm_count ? 2 : 1;
  const int vpc = 16 / split;   // n = 4 L^2 with L even: a multiple of 16
  const size_t smem = ((size_t)8 * W * (W - 1) + 16 * W + (size_t)vpc * (4 * d.k + 1)) * sizeof(cplx);
  static SmemLimit limits[3];
  void (*const fns[3])(LocalUpdateArgs, DelayedArgs) = {k_local_factors<1>, k_local_factors<2>, k_local_factors<4>};
  const int which = split == 4 ? 2 : split - 1;
  if (cudaError_t e = limits[which].raise((const void*)fns[which], (int)smem); e != cudaSuccess) return e;
  fns[which]<<<dim3(n / vpc, 2), FAC_THREADS, smem, st>>>(a, d);
  return cudaGetLastError();
}

cudaError_t launch_local_updates(const LocalUpdateArgs& a, int sm_count, cudaStream_t st, int max_grid) {
  const size_t smem = local_smem_bytes(a.mc.N);
  static SmemLimit smem_limit;
  if (cudaError_t ea = smem_limit.raise((const void*)k_local_updates, 100 * 1024); ea != cudaSuccess) return ea;
  if (smem > 100 * 1024) return cudaErrorInvalidValue;
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_local_updates, LU_THREADS, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  if (per_sm > 2) per_sm = 2;
  int grid = sm_count * per_sm;
  // small matrices: no more CTAs than warp tiles of the update
  const int n = a.mc.n;
  const int tiles = ((n + 127) / 128) * ((n + 3) / 4);
  const int need = (tiles + (LU_THREADS / 32) - 1) / (LU_THREADS / 32);
  if (grid > need) grid = need < 1 ? 1 : need;
  if (max_grid > 0 && grid > max_grid) grid = max_grid;
  LocalUpdateArgs copy = a;
  void* args[] = {&copy};
  return cudaLaunchCooperativeKernel((void*)k_local_updates, dim3(grid), dim3(LU_THREADS), args, smem, st);
}
