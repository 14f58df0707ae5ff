// Group panel of the complex-symmetric factor: as the real factors' (group_panel.cu), one dataflow launch per group of
// 64-column pivot blocks of a front -- LDL^T of each pivot block, TRSM of the rows below it, the update of the group's
// remaining columns -- with the same strips, flags and order, in complex FP64.
//
// Blocks are planar in shared memory (the real parts of 64 x 64 entries, then the imaginary ones), so a complex product is
// four FP64 tensor-core products on the real blocks' fragments. What bounds it is the chain through the pivot blocks of the
// large fronts: per block LDL^T, then the next block's rows against it and their update. The 22 launches of the edge-element
// system with 10 elements per edge (a chain of some 40 blocks) took 2.79 ms with 4 x 4 register tiles and one diagonal
// thread per four columns on the CUDA cores, now 1.17 ms; a pivot block runs only the steps of its own
// columns (1.35 ms with all eight).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../host/plan.hpp"
#include "cplx.cuh"
#include "devplan.cuh"
#include "launch.hpp"
#include "panel_blocks.cuh"
#include "pivot_steps.cuh"

namespace amp {

namespace {

constexpr int kPlane = kPanel * kPanel;  // the imaginary parts of a block follow its real parts

__device__ __forceinline__ cplx ldcg_v(const cplx *p) {
  const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
  return cplx(v.x, v.y);
}

// Complex pivot of the complex-symmetric LDL^T (ldlt.mjs:715-730): a magnitude below tau (or not a number) becomes
// tau, keeping the pivot's phase (tau itself when d = 0); a non-finite small magnitude fails the factorization.
// flags: bit 1 perturbed (a complex factor has no inertia).
__device__ __forceinline__ bool ldlt_pivot(cplx &d, double tau, int &flags) {
  flags = 0;
  const double mag = hypot(d.re, d.im);
  if (!(mag >= tau)) {
    if (!isfinite(mag)) return false;
    if (mag == 0)
      d.re = tau;
    else
      d = cplx(d.re * (tau / mag), d.im * (tau / mag));
    flags = 2;
  }
  return true;
}

// fragment of an 8 x 8 complex tile, and C += A B with K = 4 (A, B one entry per lane each, as in mma884)
struct CTile {
  double re[2], im[2];
};
__device__ __forceinline__ void cmma(CTile &c, double ar, double ai, double br, double bi) {
  mma884(c.re, ar, br);
  mma884(c.im, ar, bi);
  mma884(c.re, -ai, bi);
  mma884(c.im, ai, br);
}
__device__ __forceinline__ CTile tile_at(const double *S, int r, int c) {
  const double2 x = pair_at(S, r, c), y = pair_at(S + kPlane, r, c);
  return {{x.x, x.y}, {y.x, y.y}};
}
__device__ __forceinline__ void set_tile(double *S, int r, int c, const CTile &v) {
  set_pair(S, r, c, v.re[0], v.re[1]);
  set_pair(S + kPlane, r, c, v.im[0], v.im[1]);
}
__device__ __forceinline__ cplx at(const double *S, int r, int c) { return cplx(S[sw(r, c)], S[kPlane + sw(r, c)]); }

// c += p, p a sum of products: added to c one by one, each of a complex product's two parts would be rounded at c's size
__device__ __forceinline__ void add_tile(CTile &c, const CTile &p) {
#pragma unroll
  for (int u = 0; u < 2; u++) {
    c.re[u] += p.re[u];
    c.im[u] += p.im[u];
  }
}
// a -= b c, the product rounded by itself
__device__ __forceinline__ void csub(cplx &a, cplx b, cplx c) {
  a.re -= fma(b.re, c.re, -(b.im * c.im));
  a.im -= fma(b.re, c.im, b.im * c.re);
}

// as the real panel's load_block
__device__ __forceinline__ void load_cblock(double *S, const cplx *L, int m, int i0, int nr, int j0, int ncol, bool lower,
                                            bool pad) {
  const int lane = threadIdx.x & 31, i = 8 * (threadIdx.x >> 5) + (lane >> 2), t = lane & 3;
  cplx v[16];
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int c = 4 * e + t;
    v[e] = (i < nr && c < ncol && (!lower || c <= i)) ? ldcg_v(L + (int64_t)(j0 + c) * m + i0 + i) : cplx(0.0);
  }
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int c = 4 * e + t;
    S[sw(i, c)] = pad && i == c && i >= ncol ? 1.0 : v[e].re;
    S[kPlane + sw(i, c)] = v[e].im;
  }
}

// Pivot steps of eight columns: buffers of 64 rows x 8 columns, planar (row stride 10 as the real FP64 steps)
constexpr int kRowLd = kColLd;
constexpr int kStepPlane = kPanel * kRowLd, kStepBuf = 2 * kStepPlane;
__device__ __forceinline__ void cstep_tile(CTile &c, const double *P, const double *Q, int g, int t) {
  const double2 ar = *reinterpret_cast<const double2 *>(P + g * kRowLd + 2 * t);
  const double2 ai = *reinterpret_cast<const double2 *>(P + kStepPlane + g * kRowLd + 2 * t);
  const double2 br = *reinterpret_cast<const double2 *>(Q + g * kRowLd + 2 * t);
  const double2 bi = *reinterpret_cast<const double2 *>(Q + kStepPlane + g * kRowLd + 2 * t);
  CTile p = {{0.0, 0.0}, {0.0, 0.0}};
  cmma(p, ar.x, ai.x, br.x, bi.x);
  cmma(p, ar.y, ai.y, br.y, bi.y);
  add_tile(c, p);
}

// One pivot step for row r (eliminate8 in pivot_steps.cuh, complex). The plain form takes every pivot as it is, with
// 1 / d = conj(d) / |d|^2 from the reciprocal estimate, and returns false when a pivot of a column below w may need more:
// |d|^2 below tau2 (a little above tau^2), not a number, or out of the estimate's range; the block is then repeated with
// Exact, which perturbs (ldlt_pivot; small[k] = 1 perturbed, 2 failed) and divides. The pivots used go to piv.
template <bool Exact>
__device__ __forceinline__ bool celiminate8(const double *R, double *Pk, double *Qk, int k8, int r, int w, double tau,
                                            double tau2, cplx *piv, int *small, bool writer) {
  cplx dg[8][8], a[8];
  bool fine = true;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j <= i; j += 2) {
      const double2 x = *reinterpret_cast<const double2 *>(R + (k8 + i) * kRowLd + j);
      const double2 y = *reinterpret_cast<const double2 *>(R + kStepPlane + (k8 + i) * kRowLd + j);
      dg[i][j] = cplx(x.x, y.x);
      dg[i][j + 1] = cplx(x.y, y.y);
    }
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const double2 x = *reinterpret_cast<const double2 *>(R + r * kRowLd + j);
    const double2 y = *reinterpret_cast<const double2 *>(R + kStepPlane + r * kRowLd + j);
    a[j] = cplx(x.x, y.x);
    a[j + 1] = cplx(x.y, y.y);
  }
#pragma unroll
  for (int kk = 0; kk < 8; kk++) {
    cplx d = dg[kk][kk], iv;
    if constexpr (Exact) {
      int fl = 0;
      if (k8 + kk < w && !ldlt_pivot(d, tau, fl)) fl = 4;
      if (writer) small[k8 + kk] = fl >> 1;
      iv = cplx(1.0) / d;
    } else {
      const double n2 = fma(d.im, d.im, d.re * d.re);
      double x, f;
      const bool in = recip_parts<false>(n2, x, f);
      fine &= (in && n2 >= tau2) || k8 + kk >= w;
      const double xf = x * f;
      iv = cplx(d.re * xf, -d.im * xf);
    }
    if (writer) piv[k8 + kk] = d;
#pragma unroll
    for (int j = kk + 1; j < 8; j++) {
      const cplx lj = dg[j][kk] * iv;
#pragma unroll
      for (int i = j; i < 8; i++) {
        csub(dg[i][j], dg[i][kk], lj);
      }
      csub(a[j], a[kk], lj);
    }
    const cplx q = a[kk] * iv;
    Pk[r * kRowLd + kk] = -a[kk].re;
    Pk[kStepPlane + r * kRowLd + kk] = -a[kk].im;
    Qk[r * kRowLd + kk] = q.re;
    Qk[kStepPlane + r * kRowLd + kk] = q.im;
  }
  return fine;
}

// Pivot block: LDL^T of the 64 x 64 diagonal block, called by all 256 threads, the schedule of the real potrf_block: the
// first two warps, a row per lane, factor the eight columns' diagonal tile in registers and eliminate their rows; the
// others update the tiles of the next eight columns, hand them over, and update the rest meanwhile. Ds: the updated block
// (lower part, identity from column w on), left unchanged; scr: 11 step buffers; Lp: the block's (0, 0) entry in the front
// (ld m); Linv: the inverses of the unit L's eight 8 x 8 diagonal blocks (64 entries each, planes of 512). L = a / d with
// a unit diagonal, D to ld.D, perturbed pivots counted. On a failed pivot the status is set (first failing column
// f + c0 + k) and nothing is written.
__device__ void cpotrf_block(const double *Ds, double *scr, cplx *Lp, double *Linv, int m, int w, int f, int c0, int s,
                             unsigned long long *status, const LdltArgs<cplx> &ld) {
  __shared__ cplx piv[kPanel], scale[kPanel];
  __shared__ int small[kPanel];
  __shared__ int failAt, nPert, inexact;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, rg = row_group(warp);
  const int nk = (w + 7) >> 3;  // steps: the columns from w on are the identity's
  const double tau = ld.scal[1], tau2 = tau * tau * (1.0 + 1e-12);
  double *R = scr, *Q = R + kStepBuf, *P = R + 3 * kStepBuf;  // Q: two buffers; P: -a of every step
  const int myRow = (8 * rg + g) * kRowLd + 2 * t;
  auto hand_over = [&](const CTile &c) {
    *reinterpret_cast<double2 *>(R + myRow) = make_double2(c.re[0], c.re[1]);
    *reinterpret_cast<double2 *>(R + kStepPlane + myRow) = make_double2(c.im[0], c.im[1]);
  };
  auto panel = [&](auto exact) {  // the first two warps, a row per lane
    bool fine = true;
    for (int k = 0; k < nk; k++) {
      const int r = 8 * k + 32 * warp + lane;
      if (8 * k + 32 * warp < kPanel)
        fine &= celiminate8<decltype(exact)::value>(R, P + k * kStepBuf, Q + (k & 1) * kStepBuf, 8 * k,
                                                    min(r, kPanel - 1), w, tau, tau2, piv, small, tid == 0);
      __syncthreads();
      if (k == 0 && warp == 1) {  // row group 1's only trailing tile
        CTile c = tile_at(Ds, 8 * rg + g, 8 + 2 * t);
        cstep_tile(c, P + 8 * kRowLd, Q + 8 * kRowLd, g, t);
        hand_over(c);
      }
      __syncthreads();
    }
    if (!fine) inexact = 1;
  };
  auto trailing = [&]() {  // the other warps
    CTile c[7];            // at step k: the tiles (rg, k + 1), (rg, k + 2), ...
#pragma unroll
    for (int j = 0; j < 7; j++) {
      c[j] = {{0.0, 0.0}, {0.0, 0.0}};
      if (j < rg) c[j] = tile_at(Ds, 8 * rg + g, 8 * (j + 1) + 2 * t);
    }
    for (int k = 0; k < nk; k++) {
      __syncthreads();
      const double *Pk = P + k * kStepBuf + 8 * rg * kRowLd, *Qk = Q + (k & 1) * kStepBuf;
      if (rg > k) {
        cstep_tile(c[0], Pk, Qk + 8 * (k + 1) * kRowLd, g, t);
        hand_over(c[0]);
      }
      __syncthreads();
      if (rg > k + 1) {
#pragma unroll
        for (int j = 1; j < 7; j++) {
          if (k + 1 + j <= rg) cstep_tile(c[j], Pk, Qk + 8 * (k + 1 + j) * kRowLd, g, t);
          c[j - 1] = c[j];
        }
      }
    }
  };
  for (int pass = 0; pass < 2; pass++) {
    hand_over(tile_at(Ds, 8 * rg + g, 2 * t));
    if (tid < kPanel) small[tid] = 0;
    if (tid == 0) {
      failAt = kPanel;  // none
      nPert = inexact = 0;
    }
    __syncthreads();
    if (warp >= 2)
      trailing();
    else if (pass == 0)
      panel(std::false_type());
    else
      panel(std::true_type());
    __syncthreads();
    if (!inexact) break;  // (the second pass sets it never)
    __syncthreads();
  }
  if (tid < kPanel) {
    const int sm = tid < w ? small[tid] : 0;
    const unsigned bad = __ballot_sync(0xffffffffu, sm == 2), pert = __ballot_sync(0xffffffffu, sm == 1);
    if (lane == 0) {
      if (bad) atomicMin(&failAt, 32 * warp + __ffs(bad) - 1);
      atomicAdd(&nPert, __popc(pert));
    }
    if (tid < 8 * nk) scale[tid] = cplx(1.0) / piv[tid];
  }
  __syncthreads();
  if (failAt < kPanel) {
    if (tid == 0) atomicMin(status, status_word(f + c0 + failAt, 2, s));
    return;
  }
  if (warp >= 2) {  // the columns: a lane per row, eight columns at a time
    const int r = tid & (kPanel - 1);
    for (int p = (tid >> 6) - 1; p < 8; p += 3) {
      if (r < 8 * p || r >= w) continue;
      const double *Pr = P + p * kStepBuf + r * kRowLd;
      cplx *dst = Lp + (int64_t)(8 * p) * m + r;
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (r >= 8 * p + u)
          dst[(int64_t)u * m] = r > 8 * p + u ? cplx(-Pr[u], -Pr[kStepPlane + u]) * scale[8 * p + u] : cplx(1.0);
    }
  } else {  // column j of inv(L_pp): forward substitution with the unit block
    const int p = min(tid >> 3, nk - 1), j = tid & 7;  // (the strips use the first nk blocks)
    const double *Pp = P + p * kStepBuf + 8 * p * kRowLd;
    cplx x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      cplx v(0.0);
#pragma unroll
      for (int u = 0; u < i; u++)
        v += (cplx(Pp[i * kRowLd + u], Pp[kStepPlane + i * kRowLd + u]) * scale[8 * p + u]) * x[u];
      x[i] = i < j ? cplx(0.0) : i == j ? cplx(1.0) : v;  // (P holds -a)
      Linv[64 * p + 8 * i + j] = x[i].re;
      Linv[512 + 64 * p + 8 * i + j] = x[i].im;
    }
    // magnitudes by |re| + |im|, those of the pivots compared with by the larger part: both err towards substitution
    auto mag = [](cplx z) { return fabs(z.re) + fabs(z.im); };
    double r2 = mag(piv[8 * p + j]);  // squared norm of row j of the scaled block
#pragma unroll
    for (int u = 0; u < 7; u++) {
      const cplx a = u < j ? cplx(Pp[j * kRowLd + u], Pp[kStepPlane + j * kRowLd + u]) : cplx(0.0);
      r2 += mag(a) * mag(a * scale[8 * p + u]);
    }
    bool wild = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const double z = mag(x[i]);
      wild |= !(z * z * r2 <= kInvBound * kInvBound * fmax(fabs(piv[8 * p + i].re), fabs(piv[8 * p + i].im)));
    }
    put_wild(Linv, 2, wild);
  }
  if (tid < w) ld.D[f + c0 + tid] = piv[tid];
  if (tid == 0) atomicAdd(ld.counts + 1, nPert);
}

// C(8 x 64 of this warp) += N S^T: N the warp's A fragments (8 x 64), S a block in shared memory
__device__ __forceinline__ void cupdate_row_group(CTile (&c)[8], const CTile (&n)[8], const double *S, int g, int t) {
#pragma unroll
  for (int q = 0; q < 8; q++)
#pragma unroll
    for (int ph = 0; ph < 8; ph += 4) {
      CTile v[4];
#pragma unroll
      for (int p = 0; p < 4; p++) v[p] = tile_at(S, 8 * (ph + p) + g, 8 * q + 2 * t);
#pragma unroll
      for (int u = 0; u < 2; u++) {
#pragma unroll
        for (int p = 0; p < 4; p++) mma884(c[ph + p].re, n[q].re[u], v[p].re[u]);
#pragma unroll
        for (int p = 0; p < 4; p++) mma884(c[ph + p].im, n[q].re[u], v[p].im[u]);
#pragma unroll
        for (int p = 0; p < 4; p++) mma884(c[ph + p].re, -n[q].im[u], v[p].im[u]);
#pragma unroll
        for (int p = 0; p < 4; p++) mma884(c[ph + p].im, n[q].im[u], v[p].re[u]);
      }
    }
}

// as the real panel's substitute8, with the unit L_pp
__device__ __forceinline__ void csubstitute8(const CTile &c, CTile &w, const double *Ls, int p, int g, int t) {
  CTile x = c;
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    const double vr = __shfl_sync(0xffffffffu, k & 1 ? x.re[1] : x.re[0], 4 * g + (k >> 1));
    const double vi = __shfl_sync(0xffffffffu, k & 1 ? x.im[1] : x.im[0], 4 * g + (k >> 1));
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (2 * t + u == k) {
        w.re[u] = vr;
        w.im[u] = vi;
      }
      const cplx l = at(Ls, 8 * p + 2 * t + u, 8 * p + k);  // (nothing reads an entry after its own step)
      x.re[u] = fma(-vr, l.re, x.re[u]);
      x.re[u] = fma(vi, l.im, x.re[u]);
      x.im[u] = fma(-vr, l.im, x.im[u]);
      x.im[u] = fma(-vi, l.re, x.im[u]);
    }
  }
}

constexpr int kCGroupSmem = (3 * 2 * kPlane + 2 * 512) * (int)sizeof(double);  // one CTA per SM
static_assert(11 * kStepBuf <= 4 * kPlane, "the step buffers overlay Ls and Xs");

// The strips of one group, as k_group_panel (its comment says why no wait can deadlock). Linv: 512 complex entries per
// pivot block, two planes.
__global__ void __launch_bounds__(256, 1) k_cgroup_panel(const GroupItem *__restrict__ items,
                                                         const StripTask *__restrict__ strips, int nstrips, int *ticket,
                                                         int *flags, const __grid_constant__ DevPlan P,
                                                         cplx *__restrict__ Lx, double *__restrict__ Linv,
                                                         unsigned long long *status, LdltArgs<cplx> ld) {
  extern __shared__ __align__(16) unsigned char gp_raw[];
  double *Ls = reinterpret_cast<double *>(gp_raw);  // pivot block, rows of another diagonal strip, step buffers
  double *Xs = Ls + 2 * kPlane;                     // this strip's solved rows
  double *Ds = Xs + 2 * kPlane;                     // a diagonal strip's own pivot block
  double *Li = Ds + 2 * kPlane;                     // the pivot block's Linv
  __shared__ cplx dv[kPanel], dinv[kPanel];
  __shared__ int sTicket;
  if (threadIdx.x == 0) sTicket = factor_failed(status) ? nstrips : atomicAdd(ticket, 1);
  __syncthreads();
  const int tk = sTicket;
  if (tk >= nstrips) return;
  const StripTask st = strips[tk];
  const GroupItem it = items[st.item];
  const int s = it.s, g0 = it.g0, g1 = it.g1;
  const int f = P.snF[s], m = P.snM[s];
  const int nb = (g1 - g0 + kPanel - 1) / kPanel;
  const int r0 = st.r0, r1 = st.r1, jd = st.diag;
  const int bmax = jd >= 0 ? jd : nb;  // pivot blocks whose rows below include this strip
  const int64_t lxp = P.snLxp[s];
  cplx *L = Lx + lxp;
  int *Pf = flags + it.flag0, *Df = Pf + nb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int lr = 8 * row_group(warp) + g, row = r0 + lr;  // this lane's row of every fragment
  const bool act = row < r1;
  if (jd >= 0) load_cblock(Ds, L, m, r0, r1 - r0, r0, r1 - r0, true, true);
  CTile nx[8];  // -W of the block solved last
#pragma unroll
  for (int p = 0; p < 8; p++) nx[p] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int b = 0; b < bmax; b++) {
    const int c0 = g0 + b * kPanel, w = min(kPanel, g1 - c0);
    CTile x[8];  // the strip's rows of block b
    const cplx *src = L + (int64_t)(c0 + 2 * t) * m + row;
#pragma unroll
    for (int p = 0; p < 8; p++)
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const cplx v = act && 8 * p + 2 * t + u < w ? ldcg_v(src + (int64_t)(8 * p + u) * m) : cplx(0.0);
        x[p].re[u] = v.re;
        x[p].im[u] = v.im;
      }
    for (int q = 0; q < b; q++) {
      const int cq = g0 + q * kPanel;
      if (b > 1) {  // read the strip's W back (with one earlier block it is still in registers)
#pragma unroll
        for (int p = 0; p < 8; p++)
#pragma unroll
          for (int u = 0; u < 2; u++) {  // (every pivot block before the last of a group is full)
            const cplx v = act ? ldcg_v(ld.W + lxp + (int64_t)(cq + 8 * p + 2 * t + u) * m + row) : cplx(0.0);
            nx[p].re[u] = -v.re;
            nx[p].im[u] = -v.im;
          }
      }
      if (!panel_wait(Df + b, q + 1, status, P.spin)) return;
      if (q == 0) {  // the products are summed by themselves; after the wait's barrier nobody reads Xs any more
#pragma unroll
        for (int p = 0; p < 8; p++) {
          set_tile(Xs, lr, 8 * p + 2 * t, x[p]);
          x[p] = {{0.0, 0.0}, {0.0, 0.0}};
        }
      }
      load_cblock(Ls, L, m, c0, w, cq, kPanel, false, false);
      __syncthreads();
      cupdate_row_group(x, nx, Ls, g, t);
    }
    if (b > 0) {
#pragma unroll
      for (int p = 0; p < 8; p++) {
        const CTile v = tile_at(Xs, lr, 8 * p + 2 * t);
        add_tile(x[p], v);
      }
    }
    if (!panel_wait(Pf + b, 1, status, P.spin)) return;  // (its barrier: every warp is done with Ls)
    load_cblock(Ls, L, m, c0, w, c0, w, true, true);
    if (tid < kPanel) {
      const cplx d = tid < w ? ldcg_v(ld.D + f + c0 + tid) : cplx(1.0);
      dv[tid] = d;
      dinv[tid] = cplx(1.0) / d;
    }
    const double *Lb = Linv + ((int64_t)(it.flag0 / 2) + b) * linv_stride(2);
#pragma unroll
    for (int h = 0; h < 2; h++)
      *reinterpret_cast<double2 *>(Li + 512 * h + 2 * tid) = __ldcg(reinterpret_cast<const double2 *>(Lb + 512 * h + 2 * tid));
    const int wild = wild_blocks(Lb, 2);
    __syncthreads();
    // W = C L_bb^-T, right-looking over the 8-column blocks: solved with the block's inverse (by substitution where that is
    // large), then subtracted from the later ones
    auto solve = [&](auto some) {
#pragma unroll
      for (int p = 0; p < 8; p++) {
        if (8 * p >= w) break;  // x is zero from column w on
        CTile wv = {{0.0, 0.0}, {0.0, 0.0}};
        if (decltype(some)::value && wild >> p & 1) {
          csubstitute8(x[p], wv, Ls, p, g, t);
        } else {
          const double2 vr = *reinterpret_cast<const double2 *>(Li + 64 * p + 8 * g + 2 * t);
          const double2 vi = *reinterpret_cast<const double2 *>(Li + 512 + 64 * p + 8 * g + 2 * t);
          cmma(wv, x[p].re[0], x[p].im[0], vr.x, vi.x);
          cmma(wv, x[p].re[1], x[p].im[1], vr.y, vi.y);
        }
        x[p] = wv;
#pragma unroll
        for (int p2 = p + 1; p2 < 8; p2++) {
          if (8 * p2 >= w) break;
          const CTile l = tile_at(Ls, 8 * p2 + g, 8 * p + 2 * t);
          CTile v = {{0.0, 0.0}, {0.0, 0.0}};
          cmma(v, -wv.re[0], -wv.im[0], l.re[0], l.im[0]);
          cmma(v, -wv.re[1], -wv.im[1], l.re[1], l.im[1]);
          add_tile(x[p2], v);
        }
      }
    };
    if (wild == 0)
      solve(std::false_type());
    else
      solve(std::true_type());
    // x := L21's entries; nx := -W, W = x D
#pragma unroll
    for (int p = 0; p < 8; p++) {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int cc = 8 * p + 2 * t + u;
        const cplx xv = cplx(x[p].re[u], x[p].im[u]) * dinv[cc], wv = xv * dv[cc];
        x[p].re[u] = xv.re;
        x[p].im[u] = xv.im;
        nx[p].re[u] = -wv.re;
        nx[p].im[u] = -wv.im;
      }
      set_tile(Xs, lr, 8 * p + 2 * t, x[p]);
    }
    __syncthreads();
    for (int cc = warp; cc < w; cc += 8) {  // written column by column, a warp's lanes on consecutive rows
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = lane + 32 * h;
        if (r0 + r >= r1) continue;
        const cplx xv = at(Xs, r, cc);
        const int64_t to = (int64_t)(c0 + cc) * m + r0 + r;
        L[to] = xv;
        ld.W[lxp + to] = xv * dv[cc];
      }
    }
    if (jd < 0) continue;
    panel_release(Df + jd, b + 1);
    // the strip's own pivot block: tiles (rg, 0 .. rg) of D -= W X^T
    for (int nt = 0; nt <= lr >> 3; nt++) {
      CTile c = {{0.0, 0.0}, {0.0, 0.0}}, c2 = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const CTile v = tile_at(Xs, 8 * nt + g, 8 * q + 2 * t);
        cmma(c, nx[q].re[0], nx[q].im[0], v.re[0], v.im[0]);
        cmma(c2, nx[q].re[1], nx[q].im[1], v.re[1], v.im[1]);
      }
      CTile d = tile_at(Ds, lr, 8 * nt + 2 * t);
      add_tile(c, c2);
      add_tile(d, c);
      set_tile(Ds, lr, 8 * nt + 2 * t, d);
    }
  }
  if (jd >= 0) {  // this strip's own pivot block, fully updated: factor it and publish it (also after a failure)
    const int c0 = g0 + jd * kPanel, w = min(kPanel, g1 - c0);
    __syncthreads();  // Ds complete (also when the strip had no earlier pivot block); Ls and Xs free
    cpotrf_block(Ds, Ls, L + (int64_t)c0 * m + c0, Linv + ((int64_t)(it.flag0 / 2) + jd) * linv_stride(2), m, w, f, c0, s, status,
                 ld);
    panel_release(Pf + jd, 1);
  }
}

}  // namespace

cudaError_t init_cgroup_panel_attributes() {
  return cudaFuncSetAttribute(k_cgroup_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCGroupSmem);
}

void launch_group_panel(const GroupItem *items, const StripTask *strips, int nstrips, int *ticket, int *flags,
                        const DevPlan &P, cplx *Lx, double *Linv, unsigned long long *status, const LdltArgs<cplx> &ld,
                        cudaStream_t st) {
  if (nstrips > 0)
    k_cgroup_panel<<<(unsigned)nstrips, 256, kCGroupSmem, st>>>(items, strips, nstrips, ticket, flags, P, Lx, Linv,
                                                               status, ld);
}

}  // namespace amp
